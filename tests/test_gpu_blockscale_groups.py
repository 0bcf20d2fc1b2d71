"""Block-scale tile kernels: every K group's partial sums meet the scales of their own group, row and 128-column block, whatever
the number of groups and of accumulator buffers they go through.

The values make the results exact: operands are whole numbers of at most 2, scales are powers of two from 2^-5 to 2^5 in
the product, K is at most 11 groups.  A partial sum is a whole number of at most 512, so every sum is a multiple of 2^-5 below
11 * 512 * 2^5 < 2^18: 23 bits, nothing is ever rounded, and the outputs have to be the reference's to the last bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
E4M3 = {0: 0x00, 1: 0x38, 2: 0x40, -1: 0xB8, -2: 0xC0}


def problem(m, n, k, seed, pad=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    groups = k // 128
    table = torch.zeros(5, dtype=torch.uint8, device=DEV)
    for v, byte in E4M3.items():
        table[v + 2] = byte
    xa = torch.randint(-2, 3, (m, k), generator=g, device=DEV)
    xb = torch.randint(-2, 3, (n, k), generator=g, device=DEV)
    ea = torch.randint(-3, 4, (groups, m + pad), generator=g, device=DEV)[:, :m]
    eb = torch.randint(-2, 3, (n // 128, groups), generator=g, device=DEV)
    sfa, sfb = torch.empty((groups, m + pad), device=DEV)[:, :m], torch.exp2(eb.float())
    sfa.copy_(torch.exp2(ea.float()))
    ref = torch.zeros(m, n, dtype=torch.float64, device=DEV)
    for i in range(groups):
        part = xa[:, i * 128:(i + 1) * 128].double() @ xb[:, i * 128:(i + 1) * 128].double().t()
        ref += part * sfa[i].double()[:, None] * sfb[:, i].double().repeat_interleave(128)[None, :]
    return table[xa + 2], table[xb + 2], sfa, sfb, ref


def check(api, m, n, k, tile, flat=False, pad=0):
    a, b, sfa, sfb, ref = problem(m, n, k, m + 7 * n + k, pad)
    c = api.gemm_a8w8_blockscale(a, api.shuffle_b(b, "nk") if flat else b, sfa, sfb, out_dtype=torch.float32, tile=tile,
                                 b_flat_n=n if flat else None)
    torch.cuda.synchronize()
    assert api.last_status() == 0
    assert torch.equal(c.double(), ref)


# pair 256x256 / 256x128 / 256x224 / 256x192, one CTA 128x256 / 128x128; one group to eleven: fewer, as many and more than buffers
@pytest.mark.parametrize("tile", [4, 6, 7, 8, 2, 1])
@pytest.mark.parametrize("groups", [1, 2, 3, 4, 5, 6, 7, 11])
def test_groups_meet_their_scales(api, tile, groups):
    check(api, 333, 896, 128 * groups, tile, flat=groups % 2 == 0)


# several tiles per CTA: the buffers' phases run on from one tile to the next, ragged rows, and (4) into the column parts of tail tiles
@pytest.mark.parametrize("tile,m,n", [(4, 2309, 2048), (6, 2309, 1152), (7, 2309, 2048), (8, 2309, 1664), (2, 1601, 3328), (1, 1601, 1664)])
@pytest.mark.parametrize("groups", [4, 5])
def test_groups_across_tiles(api, tile, m, n, groups):
    check(api, m, n, 128 * groups, tile)


# 128 columns: the scales go through a ring of sixteen groups, which begins again within a tile, at a tile's end and in a shared tile's
# parts.  Rows of scales that begin anywhere.  Every sum is a multiple of 2^-5; with magnitudes that add up to less than 2^19 it takes 24 bits.
@pytest.mark.parametrize("m,n,groups", [(129, 256, 15), (129, 256, 16), (131, 256, 17), (130, 256, 37), (1, 128, 40), (1601, 1664, 18)])
@pytest.mark.parametrize("tile", [1, 0])
def test_ring_of_scales_begins_again(api, m, n, groups, tile):
    a, b, sfa, sfb, ref = problem(m, n, 128 * groups, m + groups, pad=1)
    decode = torch.zeros(256, device=DEV, dtype=torch.float64)
    for v, byte in E4M3.items():
        decode[byte] = abs(v)
    size = sum((decode[a[:, i:i + 128].long()] * sfa[i // 128].double()[:, None]) @
               (decode[b[:, i:i + 128].long()] * sfb[:, i // 128].double().repeat_interleave(128)[:, None]).t() for i in range(0, 128 * groups, 128))
    assert size.max() < 2 ** 19
    c = api.gemm_a8w8_blockscale(a, b, sfa, sfb, out_dtype=torch.float32, tile=tile)
    torch.cuda.synchronize()
    assert api.last_status() == 0
    assert torch.equal(c.double(), ref)


@pytest.mark.parametrize("tile", [4, 1])
def test_scale_rows_of_any_pitch(api, tile):
    check(api, 201, 256, 640, tile, pad=3)


# Layers back to back, operand and scales written into the same memory each time, by the quantiser directly in front of the GEMM, whose CTAs may
# be there while it writes: a warp or an epilogue that found a scale in L1 must not find what it was in the layer before.  Grids of many
# rounds, of one, and so small that a layer's CTAs come while those of the one before are still at work; rows of scales that share
# a sector with the next group's.  Against the same layers with a synchronisation after each launch.
@pytest.mark.parametrize("tile", [4, 6, 7, 8, 2, 1, 0])
@pytest.mark.parametrize("m,n,k", [(600, 768, 640), (2309, 2048, 1152), (129, 512, 512), (333, 7168, 2048)])
def test_scales_rewritten_between_layers(api, m, n, k, tile):
    g = torch.Generator(device=DEV).manual_seed(m)
    w, sfb = api.quantize_128x128(torch.randn(n, k, generator=g, device=DEV))
    xs = [torch.randn(m, k, generator=g, device=DEV, dtype=torch.bfloat16) * 4.0 ** i for i in range(6)]
    q, sfa = api.quantize_act_bf16_1x128(xs[0])

    def layers(sync):
        outs = [torch.zeros(m, n, dtype=torch.bfloat16, device=DEV) for _ in xs]
        torch.cuda.synchronize()
        for x, out in zip(xs, outs):
            api.quantize_act_bf16_1x128(x, q, sfa)
            if sync:
                torch.cuda.synchronize()
            api.gemm_a8w8_blockscale(q, w, sfa, sfb, out=out, tile=tile)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return outs

    alone, chained = layers(True), layers(False)
    assert api.last_status() == 0
    assert all(torch.equal(a, b) for a, b in zip(alone, chained))
    assert not torch.equal(alone[0], alone[1])
