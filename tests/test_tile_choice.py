"""CPU: which kernel the launcher picks, at the lines where measured times cross (148 SMs): the kind of whole tile, and how many CTAs share
a 128 x 128 tile's K where the launch takes such tiles instead."""
import ctypes as C

import pytest

from gcnasm_b200 import _lib as L


def args(m, n, k, mode=L.SCALE_NONE, hint=L.TILE_AUTO, flags=0, layout=L.B_NK_ROWMAJOR, batch=1):
    a = L.GemmArgs()
    a.ptr_a, a.ptr_b, a.ptr_c = 0x10000, 0x20000, 0x30000
    a.m, a.n, a.k, a.batch = m, n, k, batch
    a.stride_a = a.stride_b = k
    a.stride_c = n
    a.stride_a_batch, a.stride_b_batch, a.stride_c_batch = m * k, n * k, m * n
    a.scale_mode, a.tile_hint, a.flags, a.b_layout, a.out_dtype = mode, hint, flags, layout, L.OUT_BF16
    if mode in (L.SCALE_BLOCK, L.SCALE_MX):
        a.ptr_sfa, a.ptr_sfb = 0x40000, 0x50000
    if mode == L.SCALE_BLOCK:
        a.stride_sfa, a.stride_sfb = m, k // 128
    if mode == L.SCALE_MX:
        a.stride_sfa_batch, a.stride_sfb_batch = (m + 127) // 128 * (k // 128) * 512, (n + 127) // 128 * (k // 128) * 512
    return a


def choice(native, *problem, **more):
    tile = C.c_int32(-1)
    rc = native.b200_gemm_check(C.byref(args(*problem, **more)), C.byref(tile))
    return tile.value if rc == L.OK else rc


def k_split(native, *problem, bf16=False, **more):
    parts = C.c_int32(-1)
    entry = native.b200_gemm_a16w16_check_split if bf16 else native.b200_gemm_check_split
    rc = entry(C.byref(args(*problem, **more)), C.byref(parts))
    return parts.value if rc == L.OK else rc


ONE, ONE256, PAIR256, PAIR128, PAIR224 = L.TILE_128x128, L.TILE_128x256, L.TILE_PAIR_256x256, L.TILE_PAIR_256x128, L.TILE_PAIR_256x224


# a grid of one round, whole tiles: with block scales and few tiles a long K is the pair's, without scales never; 256 columns are for a short K
@pytest.mark.parametrize("mode,m,n,k,tile", [
    (L.SCALE_BLOCK, 256, 512, 512, ONE), (L.SCALE_BLOCK, 256, 512, 4096, ONE), (L.SCALE_BLOCK, 256, 512, 4224, PAIR128),
    (L.SCALE_BLOCK, 256, 512, 8192, PAIR128), (L.SCALE_BLOCK, 1024, 1024, 8192, PAIR128), (L.SCALE_BLOCK, 2048, 1024, 8192, ONE),
    (L.SCALE_NONE, 256, 512, 1024, ONE), (L.SCALE_NONE, 256, 512, 8192, ONE), (L.SCALE_NONE, 256, 8192, 8192, ONE),
    (L.SCALE_NONE, 769, 4608, 512, ONE256), (L.SCALE_NONE, 1398, 2688, 4096, ONE256), (L.SCALE_NONE, 1096, 2816, 7168, PAIR224),
    (L.SCALE_NONE, 190, 16640, 3072, ONE256), (L.SCALE_NONE, 190, 16640, 4096, PAIR256)])
def test_one_round(native, mode, m, n, k, tile):
    assert choice(native, m, n, k, mode) == tile


# few tiles with a long K: the launch splits K, whatever kind of whole tile it would take; the skinny-M kernel has its own splits
@pytest.mark.parametrize("mode,m,n,k,parts", [
    (L.SCALE_BLOCK, 256, 512, 4224, 7), (L.SCALE_BLOCK, 256, 512, 8192, 8), (L.SCALE_BLOCK, 1024, 1024, 8192, 2), (L.SCALE_BLOCK, 256, 512, 512, 1),
    (L.SCALE_NONE, 256, 512, 8192, 8), (L.SCALE_NONE, 256, 8192, 8192, 1), (L.SCALE_NONE, 256, 4608, 4096, 1), (L.SCALE_NONE, 256, 4608, 8192, 2),
    (L.SCALE_NONE, 100, 512, 8192, 8), (L.SCALE_BLOCK, 100, 512, 8192, 8), (L.SCALE_MX, 256, 512, 8192, 8),
    (L.SCALE_BLOCK, 256, 4608, 4096, 2), (L.SCALE_MX, 256, 4608, 4096, 2), (L.SCALE_NONE, 16, 512, 8192, 1), (L.SCALE_NONE, 16, 520, 8192, 8)])
def test_split_of_few_tiles(native, mode, m, n, k, parts):
    assert k_split(native, m, n, k, mode) == parts
    # inputs that are ready: a pair tile starts early and stays, a whole tile of one CTA would wait as a split one does
    early = choice(native, m, n, k, mode, flags=L.GEMM_INPUTS_READY) not in (ONE, ONE256)
    assert k_split(native, m, n, k, mode, flags=L.GEMM_INPUTS_READY) == (1 if early else parts)
    assert k_split(native, m, n, k, mode, hint=ONE) == 1                # a tile that is asked for stays whole


# few rows and 46 to 50 tiles: two CTAs a tile only where rows are whole lines apart and K is long
@pytest.mark.parametrize("m,n,k,parts", [
    (4, 6024, 5872, 1), (11, 6152, 5376, 1), (24, 6264, 8176, 1), (24, 6264, 6144, 2), (24, 6264, 6016, 1), (25, 6264, 8176, 2),
    (4, 6392, 6256, 1), (4, 6520, 6256, 2), (4, 5752, 6256, 3), (4, 6024, 8192, 2)])
def test_split_of_few_rows(native, m, n, k, parts):
    assert k_split(native, m, n, k) == parts
    assert k_split(native, m, n // 16 * 16, k // 2, bf16=True) == parts


def test_split_of_few_tiles_bf16(native):
    assert [k_split(native, *p, bf16=True) for p in ((100, 512, 4096), (256, 4608, 2048), (256, 4608, 4096), (4096, 4096, 4096))] == [8, 1, 2, 1]


# inputs that are ready: the pair kernels start before the predecessor has finished, so what they would take is not given to single CTAs
@pytest.mark.parametrize("mode", [L.SCALE_NONE, L.SCALE_TENSOR, L.SCALE_BLOCK])
@pytest.mark.parametrize("m,n,k,tile", [(1024, 1792, 1024, PAIR128), (256, 512, 1024, PAIR128), (512, 4096, 4096, PAIR128)])
def test_ready_inputs_keep_the_pair_kernels(native, mode, m, n, k, tile):
    assert choice(native, m, n, k, mode) == ONE
    assert choice(native, m, n, k, mode, flags=L.GEMM_INPUTS_READY) == tile


# MX with few tokens: the skinny-M kernel from 6 K blocks on (few tokens, or one split a panel), 12, or later with many tokens in two splits
@pytest.mark.parametrize("m,n,k,skinny", [
    (1, 512, 640, False), (1, 512, 768, True), (16, 9472, 768, True), (17, 512, 768, False), (17, 512, 1408, False), (17, 512, 1536, True),
    (64, 512, 1408, False), (64, 512, 1536, True), (64, 9600, 640, False), (64, 9600, 768, True), (32, 9472, 1536, True),
    (48, 7168, 1536, True), (64, 7168, 1536, False), (64, 7168, 2048, True), (48, 8192, 1536, False), (64, 8192, 2048, False),
    (64, 8192, 2304, True), (64, 9472, 2560, False), (64, 9472, 2688, True)])
def test_mx_few_tokens(native, m, n, k, skinny):
    assert (choice(native, m, n, k, L.SCALE_MX) == L.TILE_DECODE) == skinny
    # the same panels as batches of one quarter of the columns
    if n % 512 == 0:
        assert (choice(native, m, n // 4, k, L.SCALE_MX, batch=4) == L.TILE_DECODE) == skinny


# what b200_gemm_check reports is accepted as a hint
@pytest.mark.parametrize("mode", [L.SCALE_NONE, L.SCALE_BLOCK, L.SCALE_MX])
@pytest.mark.parametrize("layout", [L.B_NK_ROWMAJOR, L.B_FLAT_16x16])
def test_the_reported_tile_is_a_valid_hint(native, mode, layout):
    for m in (1, 16, 40, 64, 65, 200, 4096):
        for n in (512, 8192, 18432):
            for k in (256, 768, 2048, 8192):
                tile = choice(native, m, n, k, mode, layout=layout)
                assert tile > 0 and choice(native, m, n, k, mode, layout=layout, hint=tile) == tile
