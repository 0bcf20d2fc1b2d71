"""GPU: tiles of which whole chunks of columns lie behind the last one, few rows (results straight from registers): nothing is written there, and the rest is right.

Whole numbers of at most 2 and K = 128: nothing is rounded."""
import pytest
import torch

from test_gpu_tile_edges import DEV, call, whole

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,tile", [("none", 1), ("none", 2), ("none", 4), ("none", 7), ("bf16", 1), ("bf16", 2), ("bf16", 4), ("mx", 1), ("mx", 4)])
@pytest.mark.parametrize("columns", [8, 31, 32, 64, 72, 96, 127, 128, 136, 200, 224])
@pytest.mark.parametrize("m", [3, 40, 131])
def test_chunks_behind_the_last_column(api, mode, tile, columns, m):
    if tile >= 4 and m <= 128:
        m += 128                                              # a pair's second CTA then has the few rows
    n = 256 + columns
    run, ref = call(api, mode, whole(m, 128, 1), whole(n, 128, 2), tile)
    for dt in (torch.bfloat16, torch.float32):
        for extra in (256, 5):                                # pitches that 16-byte stores fit and do not fit
            wide = torch.full((m + 1, n + extra), 7.0, dtype=dt, device=DEV)
            run(wide[:m, :n])
            assert torch.equal(wide[:m, :n], ref.to(dt))
            assert torch.all(wide[:, n:] == 7.0) and torch.all(wide[m] == 7.0)
    assert api.last_status() == 0
