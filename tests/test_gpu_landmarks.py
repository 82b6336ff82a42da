"""Long runs start their tiles from landmark bounds; short ones do not. Both must give the same bits (GPU).

A run of twelve waves of source tiles or more over a strongly connected graph of out-degree 16 or more whose lengths
spread computes landmark distances first. The same sources in shorter runs take the path without: per-source summaries, histogram counts and the unrounded
fixed-point betweenness must be equal bit for bit, for weights with and without ties and over a wide range, and 32
sources' summaries must be the oracle's.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu


def graph(kind):
    c = synth.connectome(4200, 24, 0.15, weights="lognormal", seed=61, use_gpu=False, sigma=1.0)
    rng = np.random.default_rng(62)
    w = {"lognormal": c.w, "wide": np.exp2(rng.uniform(-12, 12, c.w.size)), "ties": np.exp2(rng.integers(0, 11, c.w.size))}[kind]
    assert w.mean() * (1 / w).mean() > 2
    return c.n, c.row_ptr, c.col, w


def words(a):
    """128-bit fixed-point rows as Python integers."""
    return np.array([int(lo) + (int(hi) << 64) for lo, hi in a], dtype=object)


@pytest.mark.parametrize("tile_ctas", [37, 74])  # 8 or 4 tiles in flight: 132 tiles are long, 32 short
@pytest.mark.parametrize("kind", ["lognormal", "ties", "wide"])
def test_long_and_short_runs_agree(restatement, kind, tile_ctas):
    n, rp, c, w = graph(kind)
    with ngx.Graph(n, rp, c, w) as g:
        order = g.source_order()
        kw = dict(hist_bins=128, hist_max=8.0 * float(np.median(w)), per_source=True, tile_ctas=tile_ctas)
        assert g.scc()["number_components"] == 1
        whole = g.apsp(sources=order, **kw)
        whole_bc, _ = g.brandes(sources=order, fixed=True, tile_ctas=tile_ctas)
        parts = [order[i:i + 1024] for i in range(0, n, 1024)]
        short = [g.apsp(sources=p, **kw) for p in parts]
        for k in ("sum", "sum_inv", "max", "unreachable", "arcs"):
            assert np.array_equal(whole.per_source[k], np.concatenate([r.per_source[k] for r in short])), (kind, k)
        assert np.array_equal(whole.hist, sum(r.hist for r in short)) and whole.hist_overflow == sum(r.hist_overflow for r in short)
        short_bc = sum(words(g.brandes(sources=p, fixed=True, tile_ctas=tile_ctas)[0]) for p in parts)
        assert (words(whole_bc) == short_bc).all(), kind
    want = restatement.apsp(oracle.Csr.from_arrays(n, rp, c, w), sources=order[:32])
    for k in ("sum", "sum_inv", "max"):
        assert np.array_equal(whole.per_source[k][:32], want["per_source"][k]), (kind, k)
