"""The distance phase's arc filter and its small-vertex groups, where they can go wrong (GPU, against the oracle).

Arcs are dropped when they are longer than a bound of their target's distances, in blocks of 128 arcs of one vertex, for
vertices of 16 arcs or more; smaller expansions are grouped. Distances and everything summed from them must stay bit
for bit the oracle's, betweenness within 1e-12 relative (a sum's rounding), for out-degrees around every edge, tiles
that are not full, unreachable vertices, and graphs of different sizes that take turns in one workspace slot.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu

REL = 1e-12


def graph_of_degrees(degrees, n, weights, seed):
    """Vertex i has degrees[i % len(degrees)] arcs to distinct targets."""
    rng = np.random.default_rng(seed)
    rows, cols = [0], []
    for i in range(n):
        d = min(degrees[i % len(degrees)], n - 1)
        t = rng.choice(n - 1, size=d, replace=False)
        cols.append(np.sort(np.where(t >= i, t + 1, t)))
        rows.append(rows[-1] + d)
    col = np.concatenate(cols).astype(np.int32)
    w = {"lognormal": lambda: rng.lognormal(0.0, 1.0, col.size), "int": lambda: rng.integers(1, 11, col.size).astype(np.float64),
         "wide": lambda: np.exp2(rng.uniform(-40, 40, col.size))}[weights]()
    return n, np.array(rows, np.int64), col, w


def check(result, want, label, bc=None):
    for k in ("sum_distances", "sum_inverse", "diameter", "unreachable", "reached_pairs", "traversed_arcs"):
        assert getattr(result, k) == want[k], (label, k)
    for k in ("sum", "sum_inv", "max", "unreachable", "arcs"):
        assert np.array_equal(result.per_source[k], want["per_source"][k]), (label, k)
    if bc is None:
        return
    floor = REL * max(1.0, float(np.abs(want["bc"]).mean()))
    assert (np.abs(bc - want["bc"]) <= np.maximum(REL * np.abs(want["bc"]), floor)).all(), label


def oracle_run(restatement, g):
    csr = oracle.Csr.from_arrays(*g)
    want = restatement.apsp(csr)
    want["bc"] = restatement.brandes(csr)
    return want


@pytest.mark.parametrize("weights", ["lognormal", "int", "wide"])
@pytest.mark.parametrize("degrees", [(1, 2, 3), (15, 16, 17), (31, 32, 33, 0), (127, 128, 129), (1, 255, 256, 257), (3, 300)])
def test_degrees_around_the_edges(restatement, degrees, weights):
    n, rp, c, w = graph_of_degrees(degrees, 333, weights, seed=sum(degrees))  # 333 sources: the last tile is not full
    want = oracle_run(restatement, (n, rp, c, w))
    with ngx.Graph(n, rp, c, w) as g:
        for delta in (0.0, 0.05 * w.mean(), 1e3 * w.max()):
            check(g.apsp(per_source=True, delta=delta), want, (degrees, weights, delta, "apsp"))
            bc, r = g.brandes(per_source=True, delta=delta)
            # "wide": lengths of 2^-40 vanish against distances of 2^40 (fl(d + len) == d), so equal distances join in
            # cycles, where path counts, and with them betweenness, have no value
            check(r, want, (degrees, weights, delta), bc if weights != "wide" else None)


def test_slots_shared_by_graphs_of_different_sizes(restatement):
    # dense unit-weight graphs overflow the successor lists (arc-scanning passes), larger ones follow in the same slots
    small = [synth.random_graph(300, 150, weights="unit", seed=i) for i in range(40)]
    large = [synth.random_graph(700, 18, weights="lognormal", seed=100 + i) for i in range(30)]
    graphs = [(c.n, c.row_ptr, c.col, c.w) for c in small + large]
    with ngx.Batch(graphs) as b:
        results, bcs = b.run("brandes", per_source=True, tile_ctas=1)
    assert any(r.dag_scan_tiles > 0 for r in results[: len(small)])
    for i, g in enumerate(graphs):
        if i % 7 == 0 or i >= len(small):
            check(results[i], oracle_run(restatement, g), i, bcs[i])
