"""Skinny-M kernel, the way out: 16-byte stores through shared memory, sums of K splits four columns at a time, and the element-wise
stores that ragged panels and unaligned outputs keep.

Operands are whole numbers of at most 2 and K is at most 4096, so every sum is a whole number of at most 2^14: exact in fp32, and
the fp32 output has to equal the reference; the bf16 output has to be its rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BYTES = torch.tensor([0xC0, 0xB8, 0x00, 0x38, 0x40], dtype=torch.uint8)       # e4m3 of -2 ... 2


# N: one panel, part of a warp's 32 columns (16), ragged panels, a panel count above half the SMs (no K splits); token blocks at their edges
@pytest.mark.parametrize("n,k", [(128, 256), (16, 256), (48, 128), (208, 1024), (1040, 4096), (12032, 256), (18432, 128)])
@pytest.mark.parametrize("m", [1, 15, 16, 17, 33, 64])
def test_outputs_in_both_types(api, m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * n + k)
    xa, xb = torch.randint(-2, 3, (m, k), generator=g, device=DEV), torch.randint(-2, 3, (n, k), generator=g, device=DEV)
    table = BYTES.to(DEV)
    a, b = table[xa + 2], table[xb + 2]
    ref = (xa.double() @ xb.double().t()).float()
    for dt in (torch.float32, torch.bfloat16):
        want = ref.to(dt)
        assert torch.equal(api.gemm_a8w8(a, b, out_dtype=dt), want)
        # a row pitch and a base that 16-byte stores do not fit, and what lies around C stays as it is
        wide = torch.full((m + 2, n + 5), 7.0, dtype=dt, device=DEV)
        api.gemm_a8w8(a, b, out=wide[1:m + 1, 3:n + 3])
        assert torch.equal(wide[1:m + 1, 3:n + 3], want)
        wide[1:m + 1, 3:n + 3] = 7.0
        assert torch.all(wide == 7.0)
        # a wider pitch that they do fit
        wide = torch.full((m + 2, n + 16), 7.0, dtype=dt, device=DEV)
        api.gemm_a8w8(a, b, out=wide[1:m + 1, 8:n + 8])
        assert torch.equal(wide[1:m + 1, 8:n + 8], want)
        wide[1:m + 1, 8:n + 8] = 7.0
        assert torch.all(wide == 7.0)
    assert api.last_status() == 0
