"""Betweenness on tie-free graphs, where every shortest-path DAG is a tree and dependencies are descendant counts (GPU).

The counts are integers summed from the leaves up, so betweenness must equal the oracle's exactly (every term and sum is
an integer below 2^53). Shapes where the walk can go wrong: one long chain (one walk carries on for the whole depth),
a star (one parent for every leaf), a full binary tree (every parent waits for two), combs, unreachable parts, one and
two vertices, a repeated source, tiles that are not full, groups of CTAs.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu


def from_arcs(n, arcs, seed):
    arcs = np.array(sorted(arcs), np.int64).reshape(-1, 2)
    row_ptr = np.zeros(n + 1, np.int64)
    np.add.at(row_ptr, arcs[:, 0] + 1, 1)
    return n, np.cumsum(row_ptr), arcs[:, 1].astype(np.int32), np.random.default_rng(seed).lognormal(0.0, 1.0, len(arcs))


def shape(name):
    if name == "chain":
        return from_arcs(1500, [(i, i + 1) for i in range(1499)], 1)
    if name == "star":
        return from_arcs(700, [(0, i) for i in range(1, 700)] + [(i, 0) for i in range(1, 700)], 2)
    if name == "binary":
        return from_arcs(1023, [(i, c) for i in range(511) for c in (2 * i + 1, 2 * i + 2)] + [(c, i) for i in range(511) for c in (2 * i + 1, 2 * i + 2)], 3)
    if name == "comb":
        return from_arcs(900, [(3 * i, 3 * i + 3) for i in range(299)] + [(3 * i, 3 * i + k) for i in range(300) for k in (1, 2)], 4)
    if name == "parts":
        return from_arcs(130, [(i, (i + 1) % 64) for i in range(64)] + [(64 + i, 64 + (i + 1) % 33) for i in range(33)], 5)
    if name == "one":
        return from_arcs(1, [], 6)
    if name == "two":
        return from_arcs(2, [(0, 1)], 7)
    c = synth.connectome(1111, 30, 0.15, weights="lognormal", seed=8, use_gpu=False)
    return c.n, c.row_ptr, c.col, c.w


@pytest.mark.parametrize("tile_ctas", [0, 1, 5])
@pytest.mark.parametrize("name", ["chain", "star", "binary", "comb", "parts", "one", "two", "connectome"])
def test_descendant_counts_are_exact(restatement, name, tile_ctas):
    n, rp, c, w = shape(name)
    rng = np.random.default_rng(9)
    some = np.concatenate([rng.integers(0, n, size=min(n, 45)), [0, 0]])  # repeated sources, the last tile not full
    with ngx.Graph(n, rp, c, w) as g:
        for sources in (None, some):
            want = restatement.brandes(oracle.Csr.from_arrays(n, rp, c, w), sources)
            bc, r = g.brandes(sources=sources, tile_ctas=tile_ctas)
            assert np.array_equal(bc, want), (name, tile_ctas, np.nonzero(bc != want)[0][:5])
            assert r.dag_scan_tiles == 0
