"""Grids of one round on tiles of 32 to 224 columns: 128 rows, one CTA each, the narrowest that make one round.

Operands are whole numbers of at most 2, scales powers of two from 2^-2 to 2^2 each, K at most 2688: a sum is a multiple of 2^-4 below 4 * 2688 *
2^4 < 2^18, 22 bits, so nothing is rounded and the result has to be the reference's, in bf16 its rounding.  Two rows of tiles, the second ragged; the
columns are one more than the narrower tile takes in a round, so that the last tile is ragged too and, with block scales, tiles begin
at every place of a 128-column block that the width has."""
import ctypes as C

import pytest
import torch

from gcnasm_b200 import _lib as L

from test_gpu_tile_edges import DEV, call, whole
from test_tile_choice import args

WIDTHS = [(32, 360, 384), (64, 2376, 2432), (96, 4744, 4864), (128, 7112, 7168), (160, 9480, 9600), (192, 11848, 11904), (224, 14216, 0)]


def columns(native, m, n, k, mode=L.SCALE_NONE, bf16=False, **more):
    v = C.c_int32(-1)
    assert native.b200_gemm_check_columns(C.byref(args(m, n, k, mode, **more)), int(bf16), C.byref(v)) == L.OK
    return v.value


def test_choice(native):
    for w, n, nb in WIDTHS:
        assert columns(native, 140, n, 896) == w and columns(native, 140, n, 448, bf16=True) == w
        assert columns(native, 140, nb or 14336, 896, L.SCALE_BLOCK) == (w if nb else 0)
    # the last sizes of a width and the first of the next; K for 96 and 224 columns; batches count as tiles
    assert columns(native, 100, 148 * 32, 896) == 32 and columns(native, 100, 148 * 32 + 8, 896) == 64
    assert columns(native, 140, 4744, 640) == 128 and columns(native, 140, 14216, 640) == 0 and columns(native, 140, 74 * 224 + 8, 896) == 0
    assert columns(native, 140, 360, 896, batch=7) == 64
    # several rounds without scales: 160 and 192 where they fill the last one better; a pair's tile stays where rows are not whole lines apart and K is long
    assert columns(native, 2000, 3000, 1024, bf16=True) == 192 and columns(native, 1100, 5120, 512, bf16=True) == 160
    assert columns(native, 4096, 4096, 4096, bf16=True) == 0 and columns(native, 2000, 3000, 1000, bf16=True) == 0 and columns(native, 2000, 3000, 504, bf16=True) == 192
    assert columns(native, 1200, 5120, 2048, L.SCALE_BLOCK) == 0
    assert columns(native, 776, 5504, 1152, L.SCALE_MX, batch=2) == 192 and columns(native, 776, 5504, 1280, L.SCALE_MX, batch=2) == 0
    # MX: the widths that begin at whole or half atoms of 128 columns
    assert [columns(native, 140, n, 896, L.SCALE_MX) for n in (360, 2376, 4736, 4744, 9472, 9480, 14208, 14216)] == [64, 64, 64, 128, 128, 192, 192, 0]
    # not: a tile that is asked for, K that is split, few tokens on the skinny-M kernel, inputs that are ready where the tile is a pair's
    assert columns(native, 140, 360, 896, hint=L.TILE_128x128) == 0 and columns(native, 256, 512, 8192) == 0
    assert columns(native, 64, 2432, 896) == 0
    assert columns(native, 256, 512, 1024, flags=L.GEMM_INPUTS_READY) == 0 and columns(native, 100, 512, 1024, flags=L.GEMM_INPUTS_READY) == 32


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["none", "block", "bf16"])
@pytest.mark.parametrize("w,n,nb", WIDTHS)
@pytest.mark.parametrize("kblocks", [1, 5, 6, 7, 17, 21])
def test_widths(api, mode, w, n, nb, kblocks):
    n = nb if mode == "block" else n
    if not n or (w in (96, 224) and kblocks < 6) or (w <= 64 and kblocks > 7):       # (few tiles and a long K: K is split)
        return
    m, k = 140, kblocks * (64 if mode == "bf16" else 128)
    run, ref = call(api, mode, whole(m, k, 1), whole(n, k, 2), 0)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m, n), 7.0, dtype=dt, device=DEV)
        run(out)
        assert api.last_columns() == w
        assert torch.equal(out, ref.to(dt))
        # pitches that 16-byte stores fit and do not fit; what lies around C stays as it is
        for left, extra in ((8, 16), (3, 5)):
            big = torch.full((m + 2, n + extra), 7.0, dtype=dt, device=DEV)
            run(big[1:m + 1, left:n + left])
            assert torch.equal(big[1:m + 1, left:n + left], ref.to(dt))
            big[1:m + 1, left:n + left] = 7.0
            assert torch.all(big == 7.0)
    assert api.last_status() == 0


# MX: tiles that begin in the middle of an atom, the last one with one of its two atoms or none of the second half, with every scale another
@pytest.mark.gpu
@pytest.mark.parametrize("w,m,n", [(64, 140, 360), (64, 140, 2376), (64, 200, 2440), (128, 140, 4744), (192, 140, 9480), (192, 129, 9600), (192, 140, 9696), (192, 256, 14136)])
@pytest.mark.parametrize("kblocks", [1, 2, 5, 7])
def test_mx_widths(api, w, m, n, kblocks):
    run, ref = call(api, "mx", whole(m, 128 * kblocks, 1), whole(n, 128 * kblocks, 2), 0)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m, n), 7.0, dtype=dt, device=DEV)
        run(out)
        assert api.last_columns() == w
        assert torch.equal(out, ref.to(dt))
    assert api.last_status() == 0


# several tiles per CTA: rings, accumulator buffers and the staging beside the ring run on from one to the next
@pytest.mark.gpu
@pytest.mark.parametrize("mode,w,m,n", [("bf16", 192, 2003, 3000), ("bf16", 160, 1101, 5112), ("none", 192, 574, 10180), ("none", 160, 300, 14776), ("mx", 192, 2171, 4352)])
@pytest.mark.parametrize("kblocks", [1, 3, 5, 6, 9])
def test_several_rounds(api, mode, w, m, n, kblocks):
    k = kblocks * (64 if mode == "bf16" else 128)
    run, ref = call(api, mode, whole(m, k, 1), whole(n, k, 2), 0)
    for dt in (torch.float32, torch.bfloat16):
        out = torch.full((m, n), 7.0, dtype=dt, device=DEV)
        run(out)
        assert api.last_columns() == w
        assert torch.equal(out, ref.to(dt))
    assert api.last_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["tensor", "block", "bf16"])
@pytest.mark.parametrize("w", [32, 64, 96, 128, 160, 192])
def test_flat_b_and_batches(api, kind, w):
    """Pre-shuffled B, batches (one with bf16 operands), per-tensor scales, odd rows: three or four rows of tiles in all, as many columns as
    make one round of the width and are a multiple of 128."""
    batch, m, k = (1, 257, 448) if kind == "bf16" else (2, 131, 896)
    n = 148 // (3 if kind == "bf16" else 4) * w // 128 * 128
    g = torch.Generator(device=DEV).manual_seed(w)
    a, b = (torch.randint(-2, 3, s, generator=g, device=DEV) for s in ((batch, m, k), (batch, n, k)))
    ref = torch.bmm(a.double(), b.double().transpose(1, 2))
    if kind == "bf16":
        c = api.gemm_a16w16(a[0].bfloat16(), api.shuffle_b_bf16(b[0].bfloat16(), "nk"), n=n, flat=True, out_dtype=torch.float32)[None]
    else:
        qa, qb = (torch.stack([api.cast_e4m3(x.float()) for x in t]) for t in (a, b))
        flat = torch.stack([api.shuffle_b(x, "nk") for x in qb])
        if kind == "tensor":
            s = torch.tensor([0.5], device=DEV)
            c, ref = api.flatmm_a8w8(qa, flat, n, s, s, out_dtype=torch.float32), ref * 0.25
        else:
            sfa = torch.exp2(torch.randint(-2, 3, (batch, k // 128, m), generator=g, device=DEV).float())
            sfb = torch.exp2(torch.randint(-2, 3, (batch, n // 128, k // 128), generator=g, device=DEV).float())
            c = api.gemm_a8w8_blockscale(qa, flat, sfa, sfb, b_flat_n=n, out_dtype=torch.float32)
            wa = a * sfa.transpose(1, 2).repeat_interleave(128, dim=2)
            wb = b * sfb.repeat_interleave(128, dim=1).repeat_interleave(128, dim=2)
            ref = torch.bmm(wa.double(), wb.double().transpose(1, 2))
    assert api.last_columns() == w
    assert torch.equal(c.double(), ref)
    assert api.last_status() == 0
