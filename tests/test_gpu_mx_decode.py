"""MXFP8 with few tokens: the skinny-M kernel (weights on the tensor core's M side, K split over clusters) against the oracle
and against the 128 x 128 tile kernel, which took these calls before.

Both kernels add the same fp32 products in another order: at most K/32 partial sums of one MMA each, so the difference is far
below K/32 * 2^-24 of the largest sum -- 1e-5 of max|ref| at K = 4096."""
import numpy as np
import pytest
import torch

from conftest import assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV)


# token blocks of 16, 32 and 64 at their edges; N of one slab, one panel, ragged panels, many panels; twelve K blocks, the fewest that
# more than 16 tokens in K splits go this way with, one fewer (the tile kernel), more than the ring holds
@pytest.mark.parametrize("m,n,k", [(1, 16, 1536), (16, 128, 1536), (17, 208, 1664), (32, 1040, 2048), (33, 256, 4096), (63, 4096, 1536),
                                   (64, 2064, 1664), (1, 8192, 2048), (64, 128, 4096), (64, 128, 1408)])
def test_skinny_mx(api, O, m, n, k):
    qa, ea = O.quant_mx32(O.fill_normal((m, k), 11, 0) * np.exp2(np.floor(O.fill_uniform((m, k // 32), 11, 2, -6, 6))).repeat(32, axis=1).astype(np.float32))
    qb, eb = O.quant_mx32(O.fill_normal((n, k), 11, 1) * np.exp2(np.floor(O.fill_uniform((n, k // 32), 11, 3, -6, 6))).repeat(32, axis=1).astype(np.float32))
    sa, sb = api.mx_sf_relayout(T(ea), m, k), api.mx_sf_relayout(T(eb), n, k)
    c = api.gemm_a8w8_mx(T(qa), T(qb), sa, sb, out_dtype=torch.float32).cpu().numpy()
    one = api.gemm_a8w8_mx(T(qa), T(qb), sa, sb, out_dtype=torch.float32, tile=1).cpu().numpy()
    cb = api.gemm_a8w8_mx(T(qa), T(qb), sa, sb).float().cpu().numpy()
    assert api.last_status() == 0
    ref = O.gemm_ref_mx(qa, qb, ea, eb)
    assert_close(O, c, ref, f"skinny mx {m}x{n}x{k}")
    assert np.max(np.abs(c - one)) <= 1e-5 * np.max(np.abs(ref))
    assert np.array_equal(cb, O.bf16_bits_to_f32(O.f32_to_bf16_bits(c)))


def test_skinny_mx_batched(api, O):
    """each batch reads its own atoms; ragged tokens of one batch must not meet the next one's"""
    B, m, n, k = 3, 20, 336, 1536
    parts = [(O.quant_mx32(O.fill_normal((m, k), 20 + i, 0)), O.quant_mx32(O.fill_normal((n, k), 20 + i, 1))) for i in range(B)]
    a, b = T(np.stack([p[0][0] for p in parts])), T(np.stack([p[1][0] for p in parts]))
    sa = torch.cat([api.mx_sf_relayout(T(p[0][1]), m, k) for p in parts])
    sb = torch.cat([api.mx_sf_relayout(T(p[1][1]), n, k) for p in parts])
    c = api.gemm_a8w8_mx(a, b, sa, sb, out_dtype=torch.float32).cpu().numpy()
    assert api.last_status() == 0
    for i, ((qa, ea), (qb, eb)) in enumerate(parts):
        assert_close(O, c[i], O.gemm_ref_mx(qa, qb, ea, eb), f"batch {i}")


def test_refusals_stay(api):
    from gcnasm_b200 import B200Error
    from gcnasm_b200 import _lib as L

    q = torch.zeros(16, 256, dtype=torch.uint8, device=DEV)
    w = torch.zeros(128, 256, dtype=torch.uint8, device=DEV)
    sa = torch.full((L.lib().b200_mx_sf_bytes(16, 256),), 127, dtype=torch.uint8, device=DEV)
    sb = torch.full((L.lib().b200_mx_sf_bytes(128, 256),), 127, dtype=torch.uint8, device=DEV)
    with pytest.raises(B200Error):
        api.gemm_a8w8_mx(q, w, sa, sb, tile=L.TILE_DECODE)
