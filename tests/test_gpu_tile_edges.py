"""Single-CTA tile kernels at the edges of what their ways out and their rings depend on: the rows of a tile that are there (stores from
registers or through shared memory), one tile per CTA or several (staging in the ring or beside it, its depth), the K blocks against that
depth, and with block scales the K groups against the number of scales requested ahead.

Operands are whole numbers of at most 2 and scales powers of two, K is at most 2432: a sum is a multiple of 2^-4 below 4 * 2432 * 2^4 <
2^18, 22 bits, so nothing is ever rounded.  The fp32 output has to equal the reference, the bf16 output its rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BYTES = torch.tensor([0xC0, 0xB8, 0x00, 0x38, 0x40], dtype=torch.uint8)       # e4m3 of -2 ... 2
KINDS = [("none", 1), ("none", 2), ("mx", 1), ("bf16", 1), ("bf16", 2), ("block", 1), ("block", 2)]      # tile 1: 128 x 128, 2: 128 x 256


def whole(rows, k, seed):
    return torch.randint(-2, 3, (rows, k), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


def product(xa, xb):
    return (xa.double() @ xb.double().t()).float()


def call(api, mode, xa, xb, tile):
    """(function that multiplies into an output, reference)"""
    m, k = xa.shape
    n = xb.shape[0]
    if mode == "bf16":
        a, b = xa.bfloat16(), xb.bfloat16()
        return lambda out: api.gemm_a16w16(a, b, out=out, tile=tile), product(xa, xb)
    table = BYTES.to(DEV)
    a, b = table[xa + 2], table[xb + 2]
    if mode == "mx":
        ea, eb = (127 + whole(m, k // 32, 3)).to(torch.uint8), (127 + whole(n, k // 32, 4)).to(torch.uint8)
        sa, sb = api.mx_sf_relayout(ea, m, k), api.mx_sf_relayout(eb, n, k)
        wa, wb = (x * torch.exp2(e.float() - 127).repeat_interleave(32, dim=1) for x, e in ((xa, ea), (xb, eb)))
        return lambda out: api.gemm_a8w8_mx(a, b, sa, sb, out=out, tile=tile), product(wa, wb)
    if mode == "block":
        groups = k // 128
        sfa, sfb = torch.exp2(whole(groups, m, 5).float()).contiguous(), torch.exp2(whole(n // 128, groups, 6).float()).contiguous()
        wa = xa * sfa.t().repeat_interleave(128, dim=1)
        wb = xb * sfb.repeat_interleave(128, dim=0).repeat_interleave(128, dim=1)
        return lambda out: api.gemm_a8w8_blockscale(a, b, sfa, sfb, out=out, tile=tile), product(wa, wb)
    return lambda out: api.gemm_a8w8(a, b, out=out, tile=tile), product(xa, xb)


def check(api, mode, m, n, k, tile, around=False):
    run, ref = call(api, mode, whole(m, k, 1), whole(n, k, 2), tile)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m, n), 7.0, dtype=dt, device=DEV)
        run(out)
        assert torch.equal(out, ref.to(dt)), (mode, m, n, k, tile, dt)
        if around:
            # pitches that 16-byte stores fit and do not fit; what lies around C stays as it is
            for left, extra in ((8, 16), (3, 5)):
                wide = torch.full((m + 2, n + extra), 7.0, dtype=dt, device=DEV)
                run(wide[1:m + 1, left:n + left])
                assert torch.equal(wide[1:m + 1, left:n + left], ref.to(dt))
                wide[1:m + 1, left:n + left] = 7.0
                assert torch.all(wide == 7.0)
    assert api.last_status() == 0


# rows of the last tile: one, the last and first of a warp, one to four warps; one tile and a second one below the first
@pytest.mark.parametrize("mode,tile", KINDS)
@pytest.mark.parametrize("m", [1, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 160, 161])
def test_rows_of_a_tile(api, mode, tile, m):
    check(api, mode, m, 384 if mode == "block" else 360, 256, tile, around=True)


# several tiles per CTA and ragged rows and columns
@pytest.mark.parametrize("mode,tile", KINDS)
@pytest.mark.parametrize("k", [128, 896])
def test_several_tiles_per_cta(api, mode, tile, k):
    check(api, mode, 1313, 4096 if mode == "block" else 4072, k, tile, around=True)


# K blocks (K groups with block scales): fewer, as many and more than the ring's stages (4, 6 or 7) and the scales ahead
@pytest.mark.parametrize("mode,tile", KINDS)
@pytest.mark.parametrize("kblocks", [1, 2, 3, 4, 5, 6, 7, 8, 11, 12, 13, 14, 15, 18, 19])
def test_k_blocks_against_the_ring(api, mode, tile, kblocks):
    k = kblocks * (64 if mode == "bf16" else 128)
    check(api, mode, 200, 512, k, tile)
    if kblocks in (1, 5, 6, 7, 8, 13):
        check(api, mode, 1400, 3840, k, tile)              # 330 tiles of 128 x 128, 165 of 128 x 256


# columns of the last chunk of 32 (or 16): 16-byte pieces that are whole, and single elements behind them
@pytest.mark.parametrize("mode,tile", [("none", 1), ("none", 2), ("none", 4), ("none", 6), ("none", 7), ("none", 8), ("mx", 1), ("mx", 4), ("bf16", 1), ("bf16", 2), ("bf16", 4)])
@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 9, 12, 16, 20, 23, 24, 31, 32, 33, 40, 63, 120, 250, 509])
def test_columns_of_a_chunk(api, mode, tile, n):
    check(api, mode, 140, n, 128, tile, around=True)


# block scales on 224-column pair tiles, whose chunks begin at any multiple of 16
@pytest.mark.parametrize("n", [128, 256, 384, 512, 640, 896, 1024])
def test_columns_of_a_chunk_with_block_scales(api, n):
    check(api, "block", 140, n, 256, 7, around=True)


# few rows: a stage holds what an earlier launch left behind them -- here NaNs, in every byte of every operand tile -- and nothing of it may show
@pytest.mark.parametrize("mode,tile,nan", [("none", 1, 0x7F), ("none", 2, 0x7F), ("none", 3, 0x7F), ("mx", 1, 0x7F), ("mx", 3, 0x7F), ("bf16", 1, 0xFF), ("bf16", 2, 0xFF), ("block", 3, 0x7F)])
@pytest.mark.parametrize("m", [1, 8, 17, 33, 63, 64, 65])
def test_rows_that_are_not_there(api, mode, tile, nan, m):
    if tile == 3 and m > 64:
        return
    k, n = 1792, 19200                                   # every ring goes round, every SM has a CTA
    junk = torch.full((64 if tile == 3 else 128, k), nan, dtype=torch.uint8, device=DEV)
    wide = torch.full((n, k), nan, dtype=torch.uint8, device=DEV)
    run, ref = call(api, mode, whole(m, k // 2 if mode == "bf16" else k, 1), whole(n, k // 2 if mode == "bf16" else k, 2), tile)
    if mode == "bf16":
        api.gemm_a16w16(junk.view(torch.bfloat16), wide.view(torch.bfloat16), tile=tile)
    elif mode == "mx":
        ones = [torch.full((api.mx_sf_relayout(torch.full((r, k // 32), 127, dtype=torch.uint8, device=DEV), r, k).numel(),), 127, dtype=torch.uint8, device=DEV) for r in (junk.shape[0], n)]
        api.gemm_a8w8_mx(junk, wide, *ones, tile=tile)
    elif mode == "block":
        api.gemm_a8w8_blockscale(junk, wide, torch.ones(k // 128, junk.shape[0], device=DEV), torch.ones(n // 128, k // 128, device=DEV), tile=tile)
    else:
        api.gemm_a8w8(junk, wide, tile=tile)
    out = torch.full((m, n), 7.0, device=DEV)
    run(out)
    assert torch.equal(out, ref)
    assert api.last_status() == 0


# more operands in turn than the launcher keeps tensor maps for, small sizes and addresses that differ in few bits: each call has its own
def test_many_operands_in_turn(api):
    m, n, k, count = 16, 64, 128, 300
    table = BYTES.to(DEV)
    xa, xb = whole(count * m, k, 1), whole(count * n, k, 2)
    a, b = table[xa + 2].view(count, m, k), table[xb + 2].view(count, n, k)
    ref = torch.bmm(xa.view(count, m, k).double(), xb.view(count, n, k).double().transpose(1, 2)).float()
    for _ in range(2):
        out = torch.full((count, m, n), 7.0, device=DEV)
        for i in list(range(count)) + [0, 1, 2, 0, 1, 2]:
            api.gemm_a8w8(a[i], b[i], out=out[i], tile=1 + i % 3)
        assert torch.equal(out, ref)
