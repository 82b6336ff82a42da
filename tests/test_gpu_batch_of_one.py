"""A batch of one graph gives what the graph's own handle gives (GPU).

Distances, summaries and betweenness per vertex are order-free or fixed-point sums, so they must be equal bit for bit, on a
connected graph, on one of several components and on graphs of one vertex and of none, before and after the autotuner.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
from neurograph_b200 import synth

pytestmark = pytest.mark.gpu


def graph(name):
    if name in ("one", "none"):
        n = 1 if name == "one" else 0
        return n, np.zeros(n + 1, np.int64), np.zeros(0, np.int32), np.zeros(0)
    c = synth.connectome(900, 20 if name == "connected" else 1.5, 0.15, weights="lognormal", seed=3, use_gpu=False)
    return c.n, c.row_ptr, c.col, c.w


@pytest.mark.parametrize("name", ["connected", "parts", "one", "none"])
def test_equals_the_single_handle(name):
    n, rp, col, w = graph(name)
    with ngx.Graph(n, rp, col, w) as g:
        want = g.apsp(per_source=True)
        bc_want, _ = g.brandes()
        grad_want = g.apsp_grad()[:2]
    with ngx.Batch([(n, rp, col, w)]) as b:
        for step in ("first", "replayed", "tuned"):
            if step == "tuned" and n > 0:
                b.autotune("brandes")
            (got,), _ = b.run("apsp", per_source=True, use_cuda_graph=step == "replayed")
            _, (bc,) = b.run("brandes", use_cuda_graph=step == "replayed")
            _, (grad,) = b.run("grad", use_cuda_graph=step == "replayed")
            for k in ("sum_distances", "sum_inverse", "diameter", "unreachable", "reached_pairs", "traversed_arcs"):
                assert getattr(got, k) == getattr(want, k), (step, k)
            for k, v in want.per_source.items():
                assert np.array_equal(got.per_source[k], v), (step, k)
            assert np.array_equal(bc, bc_want), step
            for a, e in zip(grad, grad_want):
                assert np.allclose(a, e, rtol=1e-12, atol=1e-13, equal_nan=True), step
