"""B200_GEMM_INPUTS_READY on each tile kernel by name: launches that may start before their predecessor has finished give the results of
launches that wait, and the last of several launches into one C wins.  (Whole numbers of at most 2: sums are exact.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BYTES = torch.tensor([0xC0, 0xB8, 0x00, 0x38, 0x40], dtype=torch.uint8)       # e4m3 of -2 ... 2


# 0: the launcher's choice; pair 256x256, 256x128, 256x224, 256x192, one CTA 128x128, 128x256
@pytest.mark.parametrize("tile", [0, 4, 6, 7, 8, 1, 2])
@pytest.mark.parametrize("block", [False, True])
@pytest.mark.parametrize("m,n,k", [(1024, 1792, 1024), (200, 512, 512)])
def test_chained_launches(api, tile, block, m, n, k):
    sets = []
    for seed in range(3):
        g = torch.Generator(device=DEV).manual_seed(seed)
        xa, xb = torch.randint(-2, 3, (m, k), generator=g, device=DEV), torch.randint(-2, 3, (n, k), generator=g, device=DEV)
        sfa, sfb = torch.ones(k // 128, m, device=DEV), torch.full((n // 128, k // 128), float(seed + 1), device=DEV)
        ref = (xa.double() @ xb.double().t()).float() * (seed + 1 if block else 1)
        sets.append((BYTES.to(DEV)[xa + 2], BYTES.to(DEV)[xb + 2], sfa, sfb, ref))

    def call(s, out):
        if block:
            api.gemm_a8w8_blockscale(*s[:4], out=out, tile=tile, inputs_ready=True)
        else:
            api.gemm_a8w8(s[0], s[1], out=out, tile=tile, inputs_ready=True)

    outs = [torch.full((m, n), 7.0, device=DEV) for _ in sets]
    shared = torch.full((m, n), 7.0, device=DEV)
    torch.cuda.synchronize()
    for _ in range(4):
        for s, out in zip(sets, outs):
            call(s, out)
        for s in sets:
            call(s, shared)
    torch.cuda.synchronize()
    assert api.last_status() == 0
    for s, out in zip(sets, outs):
        assert torch.equal(out, s[4])
    assert torch.equal(shared, sets[2][4])
