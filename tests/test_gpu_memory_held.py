"""Device memory that a handle holds (GPU): arc arrays by the stored arcs, not by the caller's; landmark rows by the budget."""

from __future__ import annotations

import gc

import numpy as np
import pytest
import torch

import neurograph_b200 as ngx
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu

SLACK = 8 << 20  # the driver maps memory in pieces of 2 MiB


def held():
    gc.collect()
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_zero_weights_take_no_arc_memory():
    """Explicit zeros are dropped: of the 56 bytes per arc (three records, a source, 4 bytes of map) only the map's 4 stay."""
    n, per_row = 4000, 2000
    m = n * per_row
    rng = np.random.default_rng(1)
    rp = np.arange(n + 1, dtype=np.int64) * per_row
    col = rng.integers(0, n, m).astype(np.int32)
    w = np.where(rng.random(m) < 0.01, rng.lognormal(0.0, 1.0, m), 0.0)
    stored = int((w != 0).sum())
    with ngx.Graph(4, np.zeros(5, np.int64), np.zeros(0, np.int32), np.zeros(0)):
        pass  # the context and the library's modules
    before = held()
    with ngx.Graph(n, rp, col, w) as g:
        assert held() - before <= 4 * m + 56 * stored + 16 * (n + 1) + SLACK
        assert g.apsp(sources=np.arange(32)).reached_pairs > 0


def test_landmark_rows_are_within_the_budget():
    """A long run over a strongly connected graph of spread lengths starts from landmark rows (512 bytes per vertex, here an
    eighth of the budget). They are part of what ngx_graph_set_memory_budget caps."""
    n = 60000
    budget = 250_000_000  # 14 slots of 17 MB without the rows
    c = synth.connectome(n, 20, 0.1, weights="lognormal", seed=5, sigma=1.0)
    with ngx.Graph(c.n, c.row_ptr, c.col, c.w) as g:
        assert g.scc()["number_components"] == 1
        sources = g.source_order()[:220 * 32]  # 220 tiles, 18 at a time
        free = g.apsp(sources=sources, per_source=True, tile_ctas=16)
    with ngx.Graph(c.n, c.row_ptr, c.col, c.w) as g:  # everything the driver loads with the first run is loaded
        before = held()
        g.set_memory_budget(budget)
        capped = g.apsp(sources=sources, per_source=True, tile_ctas=16)
        assert held() - before <= budget + SLACK
    for k, v in free.per_source.items():
        assert np.array_equal(v, capped.per_source[k]), k
