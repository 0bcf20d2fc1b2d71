"""Tiles of 32 and 64 columns whose K goes round their ring: eight stages and, with block scales, four accumulator buffers and a ring of the scales of sixteen
groups; fewer blocks than each, as many and more, K whole.

Operands are whole numbers of at most 2, scales powers of two from 2^-2 to 2^2 each, K at most 3712: a sum is a multiple of 2^-4 below 4 * 3712 * 2^4 < 2^18, 22 bits,
so nothing is rounded: the result has to be the reference's, in bf16 its rounding."""
import pytest
import torch

from test_gpu_tile_edges import BYTES, DEV, call, product, whole

pytestmark = pytest.mark.gpu
CASES = [(mode, m, n, w, kb) for mode, m, n, w, blocks in [
    ("none", 140, 360, 32, (8, 9, 15, 16, 17, 21)), ("none", 140, 2376, 64, (8, 9, 15, 16, 17, 28)), ("none", 81, 4608, 32, (29,)),
    ("bf16", 140, 360, 32, (8, 9, 15, 16, 17)), ("bf16", 140, 2376, 64, (8, 9, 15, 16, 17, 25)), ("bf16", 81, 8192, 64, (32,)),
    ("block", 140, 384, 32, (8, 9, 11, 12, 13, 15, 16, 17, 18)), ("block", 140, 2432, 64, (8, 9, 11, 12, 13, 15, 16, 17, 20)), ("block", 81, 8192, 64, (17, 29)),
    ("block", 300, 1536, 32, (21,)), ("mx", 140, 360, 64, (8, 9, 13)), ("mx", 140, 2376, 64, (8, 9, 15, 16)), ("mx", 81, 8192, 64, (17, 23))] for kb in blocks]


@pytest.mark.parametrize("mode,m,n,w,kblocks", CASES)
def test_rings_go_round(api, mode, m, n, w, kblocks):
    k = kblocks * (64 if mode == "bf16" else 128)
    run, ref = call(api, mode, whole(m, k, 1), whole(n, k, 2), 0)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m, n), 7.0, dtype=dt, device=DEV)
        run(out)
        assert api.last_columns() == w and api.last_k_split() is None
        assert torch.equal(out, ref.to(dt))
    assert api.last_status() == 0


@pytest.mark.parametrize("kind,m,n,w,kblocks", [
    ("none", 140, 384, 32, 9), ("none", 140, 384, 32, 17), ("none", 140, 2432, 64, 9), ("none", 140, 2432, 64, 17), ("bf16", 140, 384, 32, 18), ("bf16", 140, 2432, 64, 18),
    ("block", 140, 384, 32, 9), ("block", 140, 384, 32, 17), ("block", 140, 2432, 64, 9), ("block", 140, 2432, 64, 17)])
def test_rings_of_flat_b(api, kind, m, n, w, kblocks):
    k = kblocks * (64 if kind == "bf16" else 128)
    xa, xb = whole(m, k, 1), whole(n, k, 2)
    if kind == "bf16":
        c, ref = api.gemm_a16w16(xa.bfloat16(), api.shuffle_b_bf16(xb.bfloat16(), "nk"), n=n, flat=True, out_dtype=torch.float32), product(xa, xb)
    else:
        table = BYTES.to(DEV)
        a, flat = table[xa + 2], api.shuffle_b(table[xb + 2], "nk")
        if kind == "none":
            c, ref = api.flatmm_a8w8(a, flat, n, out_dtype=torch.float32), product(xa, xb)
        else:
            sfa, sfb = torch.exp2(whole(kblocks, m, 5).float()).contiguous(), torch.exp2(whole(n // 128, kblocks, 6).float()).contiguous()
            c = api.gemm_a8w8_blockscale(a, flat, sfa, sfb, b_flat_n=n, out_dtype=torch.float32)
            ref = product(xa * sfa.t().repeat_interleave(128, dim=1), xb * sfb.repeat_interleave(128, dim=0).repeat_interleave(128, dim=1))
    assert api.last_columns() == w and api.last_k_split() is None
    assert torch.equal(c, ref)
    assert api.last_status() == 0
