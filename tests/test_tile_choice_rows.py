"""How the operands' rows lie in memory decides with their sizes between one CTA's wide tiles and a pair's (148 SMs): rows that begin at whole 128-byte lines,
at whole 32-byte sectors, all of them within a line, every other one within a sector, all of them within a sector.  On the GPU each of them is compared with the
exact product (whole numbers of at most 2, scales powers of two: nothing is rounded)."""
import ctypes as C

import pytest
import torch

from gcnasm_b200 import _lib as L

from test_gpu_tile_edges import BYTES, DEV, product, whole
from test_tile_choice import args

# bytes by which rows are further apart than K, and where the operands begin
ROWS = {"lines": (0, 0), "sectors": (32, 0), "off lines": (0, 64), "half sectors": (16, 0), "no sectors": (0, 16)}
KINDS = {"none": (L.SCALE_NONE, False), "bf16": (L.SCALE_NONE, True), "block": (L.SCALE_BLOCK, False), "mx": (L.SCALE_MX, False)}


def laid_out(kind, m, n, kblocks, rows, batch=1):
    mode, bf16 = KINDS[kind]
    extra, begin = ROWS[rows]
    size = 2 if bf16 else 1
    a = args(m, n, kblocks * 128 // size, mode, batch=batch)
    a.stride_a = a.stride_b = (kblocks * 128 + extra) // size
    a.stride_a_batch, a.stride_b_batch = m * a.stride_a, n * a.stride_b
    a.ptr_a += begin
    a.ptr_b += begin
    return a


def columns(native, kind, a):
    v = C.c_int32(-1)
    assert native.b200_gemm_check_columns(C.byref(a), int(KINDS[kind][1]), C.byref(v)) == L.OK
    return v.value


# one round of `w` columns (two rows of tiles, or five) and several rounds, by K blocks: the first that are the pair's
@pytest.mark.parametrize("kind,m,n,w,first", [
    ("none", 250, 11712, 160, {"sectors": 20, "off lines": 25, "half sectors": 15, "no sectors": 15}),
    ("none", 600, 4512, 160, {"lines": None, "sectors": 20, "off lines": 25, "half sectors": 15, "no sectors": 15}),
    ("none", 250, 14144, 192, {"sectors": 10, "off lines": 16, "half sectors": 10, "no sectors": 10}),
    ("bf16", 250, 11712, 160, {"lines": None, "sectors": None, "off lines": None, "half sectors": 25, "no sectors": 25}),
    ("bf16", 600, 4512, 160, {"lines": None, "sectors": None, "off lines": None, "half sectors": 36, "no sectors": 36}),
    ("bf16", 250, 14144, 192, {"lines": None, "sectors": None, "off lines": 40, "half sectors": 15, "no sectors": 15}),
    ("bf16", 600, 5504, 192, {"lines": None, "sectors": None, "off lines": 40, "half sectors": 18, "no sectors": 18}),
    ("bf16", 250, 16512, 224, {"lines": None, "sectors": 24, "off lines": 24, "half sectors": 10, "no sectors": 10}),
    ("block", 250, 14080, 192, {"lines": None, "sectors": 41, "off lines": None, "half sectors": 41, "no sectors": 41}),
    ("mx", 600, 5504, 192, {"lines": None, "sectors": 10, "off lines": 34, "half sectors": 10, "no sectors": 16}),
    ("bf16", 1100, 5120, 160, {"lines": None, "sectors": 10, "off lines": 40, "half sectors": 10, "no sectors": 14}),
    ("bf16", 2000, 3000, 192, {"lines": None, "sectors": 10, "off lines": 17, "half sectors": 9, "no sectors": 7}),
    ("mx", 2000, 3000, 192, {"lines": 10, "sectors": 10, "off lines": 10, "half sectors": 10, "no sectors": 8})])
def test_the_pair_from_some_k_on(native, kind, m, n, w, first):
    for rows, at in first.items():
        chosen = [columns(native, kind, laid_out(kind, m, n, kb, rows)) for kb in range(6, 65)]
        assert chosen == [w if at is None or kb < at else 0 for kb in range(6, 65)], rows


def test_one_operand_or_batch_is_enough(native):
    """The worse operand decides, B that is pre-shuffled has no rows, and batches that begin elsewhere count."""
    a = laid_out("bf16", 600, 5504, 30, "lines")
    assert columns(native, "bf16", a) == 192
    for change in (lambda g: setattr(g, "ptr_a", g.ptr_a + 16), lambda g: setattr(g, "ptr_b", g.ptr_b + 48), lambda g: setattr(g, "stride_b", g.stride_b + 8)):
        a = laid_out("bf16", 600, 5504, 30, "lines")
        change(a)
        assert columns(native, "bf16", a) == 0
    a = laid_out("bf16", 600, 5504, 30, "no sectors")
    a.b_layout, a.ptr_a = L.B_FLAT_16x16, 0x10000
    assert columns(native, "bf16", a) == 192
    for batch_stride, w in ((64, 192), (8, 0)):                                     # elements: whole lines, an odd multiple of 16 bytes
        a = laid_out("bf16", 300, 4480, 30, "lines", batch=2)
        a.stride_a_batch += batch_stride
        assert columns(native, "bf16", a) == w


# rows at whole lines, 8-bit: 192 and 224 columns of two or four rows of tiles until K is long; 192 in three rounds for a pair's 224 until then, too
@pytest.mark.parametrize("m,n,w,first", [(250, 14144, 192, 28), (250, 16512, 224, 32), (500, 8224, 224, 40), (600, 5504, 192, None), (2888, 3624, 192, 10), (250, 11712, 160, None)])
def test_whole_lines_and_a_long_k(native, m, n, w, first):
    assert [columns(native, "none", laid_out("none", m, n, kb, "lines")) for kb in range(6, 65)] == [w if first is None or kb < first else 0 for kb in range(6, 65)]


# K split over CTAs against narrow whole tiles, unscaled: 64 columns of several rows of tiles for two CTAs a tile, 32 of few rows for more than four
@pytest.mark.parametrize("m,n,k,parts,w", [(2106, 312, 4608, 2, 0), (2106, 312, 4736, 2, 0), (614, 1136, 3584, 1, 64), (92, 448, 2688, 7, 0), (112, 448, 2688, 7, 0), (113, 448, 2688, 1, 32)])
def test_split_or_narrow(native, m, n, k, parts, w):
    a, v = laid_out("none", m, n, k // 128, "lines"), C.c_int32(-1)
    assert native.b200_gemm_check_split(C.byref(a), C.byref(v)) == L.OK and v.value == parts
    assert columns(native, "none", a) == w


# one row of tiles, every other row of the operands within a sector: 96 columns give way to 128 where those have two SMs a tile and K is long
@pytest.mark.parametrize("m,n,kblocks,w", [(100, 9568, 16, 96), (100, 9568, 17, 128), (100, 9728, 17, 128), (100, 9736, 17, 96)])
def test_two_sms_a_tile(native, m, n, kblocks, w):
    assert columns(native, "none", laid_out("none", m, n, kblocks, "half sectors")) == w
    assert columns(native, "none", laid_out("none", m, n, kblocks, "sectors")) == 96
    assert columns(native, "none", laid_out("none", m, n, kblocks, "no sectors")) == 96


def placed(x, extra, begin):
    """x's bytes with rows `extra` bytes further apart, in a buffer of NaNs, from `begin` bytes behind a line on"""
    rows, width = x.shape[0], x.shape[1] * x.element_size()
    buffer = torch.full((begin + rows * (width + extra),), 0xFF, dtype=torch.uint8, device=DEV)
    view = buffer[begin:].view(rows, width + extra)[:, :width]
    view.copy_(x.view(torch.uint8))
    return view.view(x.dtype) if x.dtype != torch.uint8 else view


@pytest.mark.gpu
@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("kind,m,n,kblocks", [
    ("none", 250, 11712, 14), ("none", 250, 11712, 15), ("none", 250, 14144, 10), ("none", 130, 200, 3), ("none", 100, 520, 20), ("bf16", 600, 4512, 20), ("bf16", 600, 5504, 15),
    ("bf16", 600, 5504, 18), ("bf16", 250, 16512, 10), ("bf16", 2000, 3000, 8), ("bf16", 300, 520, 7), ("block", 140, 2432, 9), ("block", 250, 14080, 3), ("mx", 600, 5504, 10),
    ("mx", 2000, 3000, 9)])
def test_products(api, native, kind, m, n, kblocks, rows):
    k = kblocks * 128 // (2 if KINDS[kind][1] else 1)
    xa, xb = whole(m, k, 1), whole(n, k, 2)
    out = torch.full((m, n), 7.0, device=DEV)
    if kind == "bf16":
        a, b = (placed(x.bfloat16(), *ROWS[rows]) for x in (xa, xb))
        ref = product(xa, xb)
        api.gemm_a16w16(a, b, out=out)
    else:
        a, b = (placed(BYTES.to(DEV)[x + 2], *ROWS[rows]) for x in (xa, xb))
        if kind == "none":
            ref = product(xa, xb)
            api.gemm_a8w8(a, b, out=out)
        elif kind == "block":
            sfa, sfb = torch.exp2(whole(kblocks, m, 5).float()).contiguous(), torch.exp2(whole(n // 128, kblocks, 6).float()).contiguous()
            ref = product(xa * sfa.t().repeat_interleave(128, dim=1), xb * sfb.repeat_interleave(128, dim=0).repeat_interleave(128, dim=1))
            api.gemm_a8w8_blockscale(a, b, sfa, sfb, out=out)
        else:
            ea, eb = (127 + whole(x.shape[0], k // 32, s) for x, s in ((xa, 3), (xb, 4)))
            ref = product(*(x * torch.exp2(e.float() - 127).repeat_interleave(32, dim=1) for x, e in ((xa, ea), (xb, eb))))
            api.gemm_a8w8_mx(a, b, api.mx_sf_relayout(ea.to(torch.uint8), m, k), api.mx_sf_relayout(eb.to(torch.uint8), n, k), out=out)
    w = columns(native, kind, laid_out(kind, m, n, kblocks, rows))
    if w:
        assert api.last_columns() == w
    assert torch.equal(out, ref)
    assert api.last_status() == 0
