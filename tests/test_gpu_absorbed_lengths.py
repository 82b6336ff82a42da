"""Betweenness and gradients where lengths vanish against distances (GPU, against a plain float64 model).

Where fl(d + len) == d, vertices at equal distances are each other's predecessors and the shortest-path DAG of a source
has cycles. The pairs on and behind such a cycle have no path count, so no dependency: the model below releases a
vertex when its last predecessor is done, in any order, and leaves the rest at 0. The library must give the model's
values (1e-12 relative: sums of the same terms in another order), and the same bits however often and after whatever
other runs in the same workspace it is asked.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle

pytestmark = pytest.mark.gpu

REL = 1e-12


def lists_graph():
    """333 vertices at out-degree 18, log-normal lengths, and a pair of arcs of 2^-60 between every tenth vertex and the next:
    both ends at one distance, a cycle; few enough DAG arcs for the successor lists."""
    rng = np.random.default_rng(3)
    n, rows, cols, ws = 333, [0], [], []
    for i in range(n):
        t = rng.choice(n, size=18, replace=False)
        t = t[(t != i) & (t != i + 1) & (t != i - 1)]
        length = rng.lognormal(0.0, 1.0, t.size)
        if i % 10 < 2 and i - i % 10 + 1 < n:
            t, length = np.append(t, i ^ 1), np.append(length, 2.0**-60)
        cols.append(t)
        ws.append(length)
        rows.append(rows[-1] + t.size)
    return n, np.array(rows, np.int64), np.concatenate(cols).astype(np.int32), np.concatenate(ws), np.arange(0, n, 3)


def scan_graph():
    """64 sources with two arcs of length 1 and a longer one each into 200 vertices joined by arcs of 2^-60: all 200 are at
    distance 1, every arc among them is a DAG arc, too many for the lists."""
    rng = np.random.default_rng(4)
    a, b = 64, 200
    rows, cols, ws = [0], [], []
    for i in range(a + b):
        t = a + rng.choice(b, size=3 if i < a else 30, replace=False)
        t = t[t != i]
        cols.append(t)
        ws.append(np.array([1.0, 1.0, 1.5]) if i < a else np.full(t.size, 2.0**-60))
        rows.append(rows[-1] + t.size)
    return a + b, np.array(rows, np.int64), np.concatenate(cols).astype(np.int32), np.concatenate(ws), np.arange(a)


def model(restatement, n, rp, col, w, sources):
    """bc per vertex and d sum(dist) / d len per arc, and the pairs that no order releases."""
    src = np.repeat(np.arange(n), np.diff(rp))
    csr = oracle.Csr.from_arrays(n, rp, col, w)
    bc, grad, stuck = np.zeros(n), np.zeros(col.size), 0
    for s in sources:
        d = restatement.sssp(csr, int(s))
        with np.errstate(invalid="ignore"):
            dag = np.nonzero(np.isfinite(d[src]) & (d[src] + w == d[col]) & (col != s))[0]
        out = [[] for _ in range(n)]
        for e in dag:
            out[src[e]].append(e)
        cnt = np.bincount(col[dag], minlength=n)
        sigma, delta = np.zeros(n), np.zeros(n)
        sigma[s] = 1.0
        order = [int(s)]
        for u in order:
            for e in out[u]:
                x = int(col[e])
                sigma[x] += sigma[u]
                cnt[x] -= 1
                if cnt[x] == 0:
                    order.append(x)
        for u in reversed(order):
            for e in out[u]:
                c = sigma[u] / sigma[col[e]] * (1.0 + delta[col[e]])
                delta[u] += c
                grad[e] += c
        delta[s] = 0.0
        bc += delta
        stuck += int((cnt > 0).sum())
    return bc, grad, stuck


def value(words):
    return np.array([int(hi) + int(lo) * 2.0**-64 for lo, hi in words])


def close(got, want):
    return (np.abs(got - want) <= REL * np.maximum(np.abs(want), max(1.0, float(np.abs(want).mean())))).all()


@pytest.mark.parametrize("tile_ctas", [1, 5])
@pytest.mark.parametrize("make", [lists_graph, scan_graph])
def test_pairs_behind_a_cycle_count_nothing(restatement, make, tile_ctas):
    n, rp, col, w, sources = make()
    bc_want, grad_want, stuck = model(restatement, n, rp, col, w, sources)
    assert stuck > 0
    with ngx.Graph(n, rp, col, w) as g:
        def run():
            bc, r = g.brandes(sources=sources, fixed=True, tile_ctas=tile_ctas)
            dcpl, deff, _ = g.apsp_grad(sources=sources, fixed=True, tile_ctas=tile_ctas)
            return bc, dcpl, deff, r.dag_scan_tiles
        first = run()
        g.apsp_grad(tile_ctas=tile_ctas)  # all sources: the workspace holds other values now
        g.brandes(sources=sources[::-1][:40], tile_ctas=tile_ctas)
        again = run()
    assert (first[3] > 0) == (make is scan_graph)
    assert close(value(first[0]), bc_want)
    assert close(value(first[1]), grad_want)
    for a, b, name in zip(first, again, ("bc", "dcpl", "deff")):
        assert np.array_equal(a, b), name
