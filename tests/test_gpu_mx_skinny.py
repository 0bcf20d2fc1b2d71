"""MXFP8 on the skinny-M kernel: the K blocks at which it takes over, pre-shuffled weights, and inputs that are ready (the weights' scale
atoms are requested before the predecessor has finished then, as the weights are).

Whole numbers of at most 2 and scales of 2^-2 to 2^2: every sum is a multiple of 2^-4 below 4 * 2304 * 2^4 < 2^18, 22 bits, so the fp32
outputs equal the reference, whatever kernel and order."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BYTES = torch.tensor([0xC0, 0xB8, 0x00, 0x38, 0x40], dtype=torch.uint8)       # e4m3 of -2 ... 2


def problem(api, m, n, k, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    whole = lambda rows, cols: torch.randint(-2, 3, (rows, cols), generator=g, device=DEV)
    xa, xb, ea, eb = whole(m, k), whole(n, k), whole(m, k // 32), whole(n, k // 32)
    full = lambda x, e: x.double() * torch.exp2(e.double()).repeat_interleave(32, dim=1)
    ref = (full(xa, ea) @ full(xb, eb).t()).float()
    table = BYTES.to(DEV)
    byte = lambda e: (127 + e).to(torch.uint8)
    return table[xa + 2], table[xb + 2], api.mx_sf_relayout(byte(ea), m, k), api.mx_sf_relayout(byte(eb), n, k), ref


def gemm(api, a, b, sa, sb, flat=False, tile=0, inputs_ready=False, out=None):
    """through the C entry: (the kernel that was reported, the result)"""
    from gcnasm_b200 import _lib as L

    m, k = a.shape
    n = b.shape[0]
    w = api.shuffle_b(b, "nk") if flat else b
    c = torch.full((m, n), 7.0, device=DEV) if out is None else out
    g = L.GemmArgs()
    g.ptr_a, g.ptr_b, g.ptr_c, g.ptr_sfa, g.ptr_sfb = a.data_ptr(), w.data_ptr(), c.data_ptr(), sa.data_ptr(), sb.data_ptr()
    g.m, g.n, g.k, g.batch = m, n, k, 1
    g.stride_a = g.stride_b = k
    g.stride_c = n
    g.scale_mode, g.out_dtype, g.tile_hint = L.SCALE_MX, L.OUT_F32, tile
    g.b_layout = L.B_FLAT_16x16 if flat else L.B_NK_ROWMAJOR
    g.flags = L.GEMM_INPUTS_READY if inputs_ready else 0
    used = C.c_int32(-1)
    assert L.lib().b200_gemm_check(C.byref(g), C.byref(used)) == L.OK
    assert L.lib().b200_gemm_a8w8(C.byref(g), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == L.OK
    if not inputs_ready:
        torch.cuda.synchronize()                       # (w may be a temporary)
        assert api.last_status() == 0
    return used.value, c


# both layouts, the three token blocks, K blocks from the fewest that are taken to more than the ring holds, with and without K splits
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 16, 768), (16, 512, 768), (17, 208, 1536), (32, 1040, 1664), (33, 256, 1792), (64, 2064, 2304), (64, 9600, 768),
                                   (5, 9616, 896), (64, 9616, 1408)])
def test_every_layout(api, flat, m, n, k):
    from gcnasm_b200 import _lib as L

    a, b, sa, sb, ref = problem(api, m, n, k, m + n + k)
    used, c = gemm(api, a, b, sa, sb, flat)
    assert used == L.TILE_DECODE
    assert torch.equal(c, ref)
    used, c = gemm(api, a, b, sa, sb, flat, tile=L.TILE_128x128)
    assert used == L.TILE_128x128 and torch.equal(c, ref)


# both sides of each line: the kernel that is not the launcher's choice gives the same sums
@pytest.mark.parametrize("m,n,k", [(16, 512, 640), (17, 512, 1408), (64, 512, 1408), (64, 8192, 2048), (64, 8192, 2304), (40, 8192, 1536), (64, 9600, 640)])
def test_both_sides_of_a_line(api, m, n, k):
    from gcnasm_b200 import _lib as L

    a, b, sa, sb, ref = problem(api, m, n, k, 5)
    for tile in (0, L.TILE_128x128) + ((L.TILE_DECODE,) if k >= 768 else ()):
        assert torch.equal(gemm(api, a, b, sa, sb, tile=tile)[1], ref)


def test_ready_inputs(api):
    sets = [problem(api, 16, 2048, 2048, s) for s in range(3)]
    outs = [torch.full_like(s[4], 7.0) for s in sets]
    shared = torch.full_like(outs[0], 7.0)
    torch.cuda.synchronize()
    for _ in range(4):
        for s, o in zip(sets, outs):
            gemm(api, *s[:4], inputs_ready=True, out=o)
        for s in sets:
            gemm(api, *s[:4], inputs_ready=True, out=shared)
    torch.cuda.synchronize()
    assert api.last_status() == 0
    for s, o in zip(sets, outs):
        assert torch.equal(o, s[4])
    assert torch.equal(shared, sets[2][4])             # consecutive launches into one C: the last one wins
