"""128 x 128 tiles whose K is split over a cluster: few tiles and a long K.

Without scales, with block scales and with bf16 operands the values are whole numbers (of at most 2, block scales 2^-5 to 2^5 in the
product): an fp32 sum of at most 8192 products, or of scaled groups in steps of 2^-5 whose magnitudes sum to less than 2^19 (checked), takes 24
bits, nothing is rounded, and the result has to be the exact one.  MX: a sum of K products in any order and grouping is off by at most
K * 2^-23 of the sum of their magnitudes.  Every test holds how many CTAs shared a tile in its launch."""
import ctypes as C
import os
import subprocess

import pytest
import torch

from gcnasm_b200 import _lib as L

from test_gpu_blockscale_groups import problem
from test_tile_choice import args

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# CTAs per tile, batches, rows, columns, K: every count, tiles of one row and with a ragged edge each way, an odd number of K blocks (a shorter last part)
SHAPES = [(8, 2, 100, 512, 4096), (8, 2, 1, 136, 8192), (8, 1, 1, 136, 8192), (7, 2, 129, 264, 4224), (7, 1, 129, 768, 4224), (6, 1, 130, 1280, 8192),
          (5, 1, 200, 1536, 8192), (4, 1, 256, 2048, 3968), (4, 1, 384, 768, 4096), (3, 1, 120, 5120, 8192), (3, 1, 45, 5000, 8192), (2, 1, 256, 4608, 8192)]


def ints(g, *shape):
    return torch.randint(-2, 3, shape, generator=g, device=DEV)


@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("kind", ["fp8", "tensor", "bf16"])
@pytest.mark.parametrize("parts,batch,m,n,k", SHAPES)
def test_sums_are_exact(api, kind, parts, batch, m, n, k, flat, out):
    if flat:
        n = (n + 15) // 16 * 16
        m = max(m, 65) if kind != "bf16" else m                 # (8-bit operands, fewer rows and 16-column blocks: the skinny-M kernel)
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    if kind == "bf16":
        batch, k = 1, k // 2
    a, b = ints(g, batch, m, k), ints(g, batch, n, k)
    ref = torch.bmm(a.double(), b.double().transpose(1, 2))
    if kind == "bf16":
        w = b[0].bfloat16()
        c = api.gemm_a16w16(a[0].bfloat16(), api.shuffle_b_bf16(w, "nk") if flat else w, n=n, flat=flat, out_dtype=out)
    else:
        qa, qb = (torch.stack([api.cast_e4m3(t[i].float()) for i in range(batch)]) for t in (a, b))
        s = torch.tensor([0.5], device=DEV) if kind == "tensor" else None
        ref = ref * 0.25 if kind == "tensor" else ref
        if flat:
            c = api.flatmm_a8w8(qa, torch.stack([api.shuffle_b(qb[i], "nk") for i in range(batch)]), n, s, s, out_dtype=out)
        else:
            c = api.gemm_a8w8(qa, qb, s, s, out_dtype=out)
    assert api.last_k_split() == parts
    torch.cuda.synchronize()
    assert api.last_status() == 0
    assert torch.equal(c.reshape(batch, m, n), ref.float().to(out))


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("parts,m,n,groups", [(8, 100, 512, 32), (7, 333, 512, 33), (8, 129, 128, 23), (2, 256, 4608, 32), (3, 120, 5120, 31), (4, 200, 2048, 40),
                                              (5, 200, 1536, 64), (6, 130, 1280, 61)])
def test_groups_meet_their_scales(api, parts, m, n, groups, flat):
    a, b, sfa, sfb, ref = problem(m, n, 128 * groups, m + groups)
    magnitudes = (a.view(torch.float8_e4m3fn).double().abs() * sfa.double().t().repeat_interleave(128, 1)) @ (
        b.view(torch.float8_e4m3fn).double().abs() * sfb.double().repeat_interleave(128, 0).repeat_interleave(128, 1)).t()
    assert magnitudes.max() < 2 ** 19
    c = api.gemm_a8w8_blockscale(a, api.shuffle_b(b, "nk") if flat else b, sfa, sfb, out_dtype=torch.float32, b_flat_n=n if flat else None)
    assert api.last_k_split() == parts
    torch.cuda.synchronize()
    assert api.last_status() == 0
    assert torch.equal(c.double(), ref)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("parts,m,n,k", [(8, 100, 512, 4096), (7, 129, 768, 4224), (6, 130, 1280, 8192), (5, 200, 1536, 8192), (4, 256, 2048, 3968),
                                         (3, 120, 5120, 8192), (2, 256, 4608, 4096), (7, 129, 264, 4224)])
def test_mx(api, parts, m, n, k, flat):
    n = (n + 15) // 16 * 16 if flat else n
    g = torch.Generator(device=DEV).manual_seed(m)
    sides = []
    for rows in (m, n):
        q, logical, atoms = api.quantize_mx32(torch.randn(rows, k, generator=g, device=DEV))
        value = q.view(torch.float8_e4m3fn).double() * torch.exp2(logical.reshape(rows, -1).double() - 127).repeat_interleave(32, 1)
        sides.append((q, atoms, value))
    (a, sfa, va), (b, sfb, vb) = sides
    if flat:
        c = api._gemm(a, api.shuffle_b(b, "nk"), n=n, sfa=sfa, sfb=sfb, scale_mode=L.SCALE_MX, b_layout=L.B_FLAT_16x16, out_dtype=torch.float32)
    else:
        c = api.gemm_a8w8_mx(a, b, sfa, sfb, out_dtype=torch.float32)
    assert api.last_k_split() == parts
    torch.cuda.synchronize()
    assert api.last_status() == 0
    assert ((c.double() - va @ vb.t()).abs() <= k * 2.0 ** -23 * (va.abs() @ vb.abs().t())).all()


def test_captured_behind_the_kernel_that_writes_b(api):
    """A CUDA graph of shuffle and GEMM: B and A come anew before each replay, and the GEMM is launched while the shuffle still writes."""
    m, n, k = 100, 1280, 8192
    g = torch.Generator(device=DEV).manual_seed(9)
    a, b = api.cast_e4m3(ints(g, m, k).float()), api.cast_e4m3(ints(g, n, k).float())
    out, stream, graph = torch.zeros(m, n, device=DEV), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    api.flatmm_a8w8(a, api.shuffle_b(b, "nk"), n, out=out)
    assert api.last_k_split() == 8
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        api.flatmm_a8w8(a, api.shuffle_b(b, "nk"), n, out=out)
    assert api.last_k_split() == 8
    for _ in range(3):
        x, y = ints(g, m, k), ints(g, n, k)
        a.copy_(api.cast_e4m3(x.float()))
        b.copy_(api.cast_e4m3(y.float()))
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.double(), x.double() @ y.double().t())
    assert api.last_status() == 0


@pytest.mark.parametrize("mode", [L.SCALE_NONE, L.SCALE_BLOCK, L.SCALE_MX])
@pytest.mark.parametrize("m,n,k", [(256, 4608, 8192), (100, 5120, 8192), (256, 2048, 4096), (200, 1536, 8192), (100, 512, 512), (256, 512, 8192)])
def test_the_launch_is_the_reported_one(api, native, mode, m, n, k):
    a, b = (torch.zeros(rows, k, dtype=torch.uint8, device=DEV) for rows in (m, n))
    run = {L.SCALE_NONE: lambda: api.gemm_a8w8(a, b),
           L.SCALE_BLOCK: lambda: api.gemm_a8w8_blockscale(a, b, torch.ones(k // 128, m, device=DEV), torch.ones(n // 128, k // 128, device=DEV)),
           L.SCALE_MX: lambda: api.gemm_a8w8_mx(a, b, *(torch.full((native.b200_mx_sf_bytes(rows, k),), 127, dtype=torch.uint8, device=DEV)
                                                        for rows in (m, n)))}[mode]
    run()
    parts = C.c_int32(-1)
    assert native.b200_gemm_check_split(C.byref(args(m, n, k, mode)), C.byref(parts)) == 0
    assert (api.last_k_split() or 1) == parts.value
    api.gemm_a8w8(a[:, :128].contiguous(), b[:, :128].contiguous())             # a launch of whole tiles
    assert api.last_k_split() is None
    torch.cuda.synchronize()
    assert api.last_status() == 0


def test_driver_names_the_tile_it_launches(native):
    from gcnasm_b200 import build

    build.build_drivers()
    out = subprocess.run([os.path.join(build.BIN, "gemm_a8w8_blockscale"), "-m", "256", "-n", "512", "-k", "8192", "-b", "1", "--warmup", "1", "--iters", "1"],
                         capture_output=True, text=True, timeout=300).stdout
    assert "tile_config=1, k_split=8" in out


# who names a 128 x 128 tile gets it whole: the bits of every other kind of whole tile
@pytest.mark.parametrize("m,n,k", [(200, 512, 4096), (333, 384, 8192)])
def test_a_tile_that_is_asked_for_stays_whole(api, m, n, k):
    g = torch.Generator(device=DEV).manual_seed(k)
    (a, sfa), (b, sfb) = (q(torch.randn(rows, k, generator=g, device=DEV)) for q, rows in ((api.quantize_1x128, m), (api.quantize_128x128, n)))
    for run in (lambda t: api.gemm_a8w8(a, b, out_dtype=torch.float32, tile=t),
                lambda t: api.gemm_a8w8_blockscale(a, b, sfa, sfb, out_dtype=torch.float32, tile=t)):
        pair, one = run(6), run(1)
        assert api.last_k_split() is None
        assert torch.equal(pair, one)
    x, y = (torch.randn(rows, k // 2, generator=g, device=DEV).bfloat16() for rows in (m, n))
    assert torch.equal(api.gemm_a16w16(x, y, out_dtype=torch.float32, tile=4), api.gemm_a16w16(x, y, out_dtype=torch.float32, tile=1))
    torch.cuda.synchronize()
    assert api.last_status() == 0


def test_strided_result_in_a_chain(api):
    """Rows of C further apart than N and not 16-byte aligned, behind the kernel that writes A."""
    g = torch.Generator(device=DEV).manual_seed(3)
    m, n, k = 200, 272, 4096
    b = ints(g, n, k)
    qb = api.cast_e4m3(b.float())
    for i in range(3):
        a = ints(g, m, k)
        big = torch.full((m, n + 3), 7.0, device=DEV)
        api.gemm_a8w8(api.cast_e4m3(a.float()), qb, out=big[:, 1:n + 1])
        assert api.last_k_split() == 8
        torch.cuda.synchronize()
        assert torch.equal(big[:, 1:n + 1].double(), a.double() @ b.double().t())
        assert (big[:, 0] == 7).all() and (big[:, n + 1:] == 7).all()
