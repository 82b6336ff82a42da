"""The default bucket width on both sides of its rule's lines changes the work, never the results (GPU).

The rule doubles the width below a mean out-degree of 32 and below a length spread of 2. Per source, sums and maxima of
distances and of inverse distances must be the oracle's, and betweenness within its 1e-12.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["wide", "narrow", "equal"])
@pytest.mark.parametrize("degree", [1, 31, 32, 33])
def test_default_width_keeps_results(restatement, degree, weights):
    n = 333
    rng = np.random.default_rng(degree)
    col = np.concatenate([rng.choice(n, degree, replace=False) for _ in range(n)]).astype(np.int32)
    rp = (np.arange(n + 1) * degree).astype(np.int64)
    w = {"wide": np.exp(rng.normal(0.0, 1.2, col.size)), "narrow": rng.integers(4, 8, col.size).astype(np.float64), "equal": np.full(col.size, 0.7)}[weights]
    assert (w.mean() * (1 / w).mean() < 2) == (weights != "wide")
    csr = oracle.Csr.from_arrays(n, rp, col, w)
    want, bc_want = restatement.apsp(csr), restatement.brandes(csr)
    with ngx.Graph(n, rp, col, w) as g:
        got = g.apsp(per_source=True)
        bc, _ = g.brandes()
    for k in ("sum", "sum_inv", "max"):
        assert np.array_equal(got.per_source[k], want["per_source"][k]), k
    assert np.allclose(bc, bc_want, rtol=1e-12, atol=1e-12 * max(1.0, float(np.abs(bc_want).mean())))
