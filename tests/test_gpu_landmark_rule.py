"""Runs whose caller sets a large group size start from landmark bounds at 128 tiles, not at twelve waves of a few (GPU).

With 74 CTAs per tile twelve waves are 48 tiles, too few to pay for the two landmark tiles. Whether a run had them shows in
the memory of their rows (512 bytes per vertex), which stays with the handle until a run without.
"""

from __future__ import annotations

import gc

import pytest
import torch

import neurograph_b200 as ngx
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu


def held():
    gc.collect()
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("tiles,rows", [(127, False), (128, True)])
def test_rows_are_computed_from_128_tiles_on(tiles, rows):
    n = 60000
    c = synth.connectome(n, 24, 0.1, weights="lognormal", seed=5, sigma=1.0)
    with ngx.Graph(c.n, c.row_ptr, c.col, c.w) as g:
        assert g.scc()["number_components"] == 1
        sources = g.source_order()[:tiles * 32]
        g.apsp(sources=sources, tile_ctas=74, max_iterations=1 << 40)  # an iteration limit rules them out
        without = held()
        g.apsp(sources=sources, tile_ctas=74)
        assert (held() - without > 256 * n) == rows
