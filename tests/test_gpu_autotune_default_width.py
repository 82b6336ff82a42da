"""The default bucket width at its rule's line, and among the autotuner's trials (GPU).

Untuned runs double the width below a mean out-degree of 28, which changes no result. On a ring of equal lengths a search has one pending vertex per source, so a bucket costs one step whatever its width, and
wider is faster: the default of four lengths by 14 % over the widest of the fixed multiples.
"""

from __future__ import annotations

import numpy as np
import pytest

import neurograph_b200 as ngx
import oracle

pytestmark = pytest.mark.gpu


def test_the_default_width_is_tried():
    n = 3000
    with ngx.Graph(n, np.arange(n + 1, dtype=np.int64), ((np.arange(n) + 1) % n).astype(np.int32), np.full(n, 2.0)) as g:
        assert g.autotune("apsp")["delta_scale"] == 4.0


@pytest.mark.parametrize("degree", [27, 28, 29])
def test_widths_around_the_line_give_the_same_results(restatement, degree):
    n = 333
    rng = np.random.default_rng(degree)
    col = np.concatenate([rng.choice(n, degree, replace=False) for _ in range(n)]).astype(np.int32)
    rp = (np.arange(n + 1) * degree).astype(np.int64)
    w = rng.lognormal(0.0, 1.2, col.size)
    assert w.mean() * (1 / w).mean() > 2
    want = restatement.apsp(oracle.Csr.from_arrays(n, rp, col, w))
    with ngx.Graph(n, rp, col, w) as g:
        got = g.apsp(per_source=True)
    for k in ("sum", "sum_inv", "max"):
        assert np.array_equal(got.per_source[k], want["per_source"][k]), k
