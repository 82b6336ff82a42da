"""Workloads of the all-sources shortest-path library, from the smallest call to the largest, through its public API.

Every graph is a seeded synthetic connectome of the shape the reference is used on: vertices uniform in the unit cube,
out-degree Poisson(degree), targets at distances drawn from exp(-r / length_scale) (or uniform targets: "uniform"),
no repeated arcs, FP64 weights: integers 1..10 (many equal path lengths), log-normal(0, sigma) or unit.

A program that uses the library builds a graph handle once and then asks it for metrics, so the handle is part of the
prepared state; only the differentiable form builds its handle inside the pass, because its public function does.
"""

import math

import numpy as np
import torch

from neurograph_b200 import Batch, Graph
from neurograph_b200.autograd import apsp_metrics

HIST_BINS = 1024  # the distance histogram's size in the library's benchmark


def listed():
    return [
        # the smallest call: one small circuit, all sources, where launches and the host path count
        {"name": "apsp_small", "kind": "apsp", "n": 300, "degree": 8.0, "scale": 0.2, "weights": "lognormal", "sigma": 1.0, "sources": 0, "hist": 64},
        # distance rows of a few seeds, handed to the caller (a seed-based analysis)
        {"name": "rows_seeds", "kind": "rows", "n": 20011, "degree": 20.0, "scale": 0.1, "weights": "lognormal", "sigma": 1.0, "sources": 50, "hist": 0},
        # the plain small configuration: sparse, integer weights, every metric of a run (APSP, histogram, betweenness)
        {"name": "brandes_sparse_int", "kind": "brandes", "n": 5000, "degree": 6.0, "scale": 0.1, "weights": "int", "sigma": 0.0, "sources": 0, "hist": HIST_BINS},
        # integer weights at a connectome's density: shortest paths tie often
        {"name": "brandes_ties", "kind": "brandes", "n": 10007, "degree": 40.0, "scale": 0.1, "weights": "int", "sigma": 0.0, "sources": 0, "hist": HIST_BINS},
        # inverse-weight metric on a fragmented graph (many strongly connected components, unreachable pairs)
        {"name": "apsp_inverse_fragments", "kind": "apsp_inverse", "n": 20011, "degree": 2.0, "scale": 0.0, "weights": "uniform", "sigma": 1.0, "sources": 0, "hist": 0},
        # strongly connected components of a large sparse connectome: one giant component and a fringe of small ones
        {"name": "scc", "kind": "scc", "n": 300000, "degree": 4.0, "scale": 0.08, "weights": "lognormal", "sigma": 1.0, "sources": 0, "hist": 0},
        # a cohort: many graphs of mixed size and weight kind in one batch, betweenness for all of them
        {"name": "batch_cohort", "kind": "batch", "n": 6000, "degree": 32.0, "scale": 0.1, "weights": "mixed", "sigma": 1.0, "graphs": 24, "sources": 0, "hist": HIST_BINS},
        # one optimisation step on the weights of a small model: metrics forward, gradient backward
        {"name": "train_step", "kind": "train", "n": 2000, "degree": 20.0, "scale": 0.15, "weights": "lognormal", "sigma": 0.5, "sources": 0, "hist": 0},
        # the adjoint on a mid-size connectome: weights updated in place, metrics and their gradients for a block of sources
        {"name": "grad_mid", "kind": "grad", "n": 50000, "degree": 40.0, "scale": 0.08, "weights": "lognormal", "sigma": 0.5, "sources": 2048, "hist": 0},
        # the batched single-graph configuration: a block of the all-sources order, distances and histogram
        {"name": "apsp_large", "kind": "apsp", "n": 100000, "degree": 100.0, "scale": 0.08, "weights": "lognormal", "sigma": 1.0, "sources": 4736, "hist": HIST_BINS},
        # the same graph with betweenness: the headline workload
        {"name": "brandes_large", "kind": "brandes", "n": 100000, "degree": 100.0, "scale": 0.08, "weights": "lognormal", "sigma": 1.0, "sources": 2368, "hist": HIST_BINS},
        # the largest graph of the configurations: a sample of its sources
        {"name": "brandes_million", "kind": "brandes", "n": 1000000, "degree": 40.0, "scale": 0.05, "weights": "lognormal", "sigma": 1.0, "sources": 512, "hist": HIST_BINS},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apsp", "apsp", "brandes", "brandes", "brandes", "grad", "apsp_inverse", "rows", "scc", "train", "batch"])
    weights = rng.choice(["int", "lognormal", "lognormal", "unit"])
    sigma = rng.choice([0.5, 1.0])
    if kind == "batch":
        return {"kind": "batch", "n": _log_int(rng, 500, 6000), "degree": round(math.exp(rng.uniform(math.log(5), math.log(40))), 2), "scale": 0.1,
                "weights": "mixed", "sigma": 1.0, "graphs": rng.randint(3, 24), "sources": 0, "hist": rng.choice([0, HIST_BINS])}
    n = _log_int(rng, 300, 3000) if kind == "train" else _log_int(rng, 300, 300000)
    if kind == "train" and weights == "unit":
        weights = "lognormal"
    degree = round(math.exp(rng.uniform(math.log(5), math.log(100))), 2)
    if kind == "apsp_inverse":
        weights = "uniform"
        degree = round(rng.uniform(1.5, 12.0), 2)
    degree = min(degree, n / 6)
    # all sources where that is affordable, else a block of the all-sources order (a ragged count, at most about 1e10
    # (source, arc) pairs)
    most = int(1.0e10 / (n * degree))
    sources = 0 if most >= n and rng.random() < 0.8 else min(_log_int(rng, 20, 3000), n, max(20, most))
    if kind == "rows":
        sources = min(_log_int(rng, 1, 200), n, max(1, int(2.0e7 / n)))
    if kind in ("train", "scc"):
        sources = 0
    if kind == "scc":
        degree = round(rng.uniform(1.5, 6.0), 2)
    hist = rng.choice([0, 100, HIST_BINS]) if kind in ("apsp", "brandes") else 0
    scale = 0.0 if kind == "apsp_inverse" and rng.random() < 0.5 else round(rng.uniform(0.05, 0.2), 3)
    return {"kind": kind, "n": n, "degree": degree, "scale": scale, "weights": weights, "sigma": sigma, "sources": sources, "hist": hist}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _csr(n, degree, scale, weights, sigma, seed):
    """One seeded graph as host arrays (row_ptr, col, w)."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    # more arcs than asked for: repeated ones are dropped, then as many as leave round(n * degree) of them
    want = int(round(n * degree))
    deg = torch.poisson(torch.full((n,), float(degree) * (1.15 if n > 4000 else 2.0), device=dev), generator=gen).to(torch.int64)
    src = torch.repeat_interleave(torch.arange(n, device=dev), deg)
    m = int(src.numel())
    if scale > 0.0:
        # the target is a vertex of the grid cell that a displacement of density r^2 exp(-r / scale) ends in
        side = max(1, int((n / 4) ** (1 / 3)))
        pos = torch.rand(n, 3, device=dev, generator=gen)
        cell = (pos * side).to(torch.int64).clamp_(0, side - 1)
        cell = (cell[:, 0] * side + cell[:, 1]) * side + cell[:, 2]
        by_cell = torch.sort(cell, stable=True).indices
        count = torch.bincount(cell, minlength=side**3)
        start = torch.cumsum(count, 0) - count
        r = -scale * torch.log(torch.rand(m, 3, device=dev, generator=gen).clamp_(min=1e-12)).sum(1)
        dirs = torch.randn(m, 3, device=dev, generator=gen)
        dirs = dirs / dirs.norm(dim=1, keepdim=True).clamp_(min=1e-12)
        p = pos[src] + r[:, None] * dirs
        p = (1 - (1 - p.abs()).abs()).clamp_(0, 1)
        c = (p * side).to(torch.int64).clamp_(0, side - 1)
        c = (c[:, 0] * side + c[:, 1]) * side + c[:, 2]
        pick = (torch.rand(m, device=dev, generator=gen) * count[c]).to(torch.int64)
        dst = by_cell[(start[c] + pick).clamp_(max=n - 1)]
        del r, dirs, p, c, pick
    else:
        dst = (torch.rand(m, device=dev, generator=gen, dtype=torch.float64) * n).to(torch.int64).clamp_(max=n - 1)
    key = torch.unique((src * n + dst)[src != dst])
    if key.numel() > want:
        key = key[torch.sort(torch.randperm(key.numel(), device=dev, generator=gen)[:want]).values]
    src, dst = key // n, key % n
    m = int(key.numel())
    if weights == "int":
        w = torch.randint(1, 11, (m,), device=dev, generator=gen).to(torch.float64)
    elif weights == "lognormal":
        w = torch.exp(sigma * torch.randn(m, device=dev, generator=gen, dtype=torch.float64))
    elif weights == "uniform":
        w = 0.1 + 9.9 * torch.rand(m, device=dev, generator=gen, dtype=torch.float64)
    else:
        w = torch.ones(m, device=dev, dtype=torch.float64)
    row_ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return row_ptr.cpu().numpy(), dst.to(torch.int32).cpu().numpy(), w.cpu().numpy()


def _batch_shapes(case):
    """Sizes of the cohort's graphs (the same for every seed): up to case["n"] vertices, mixed densities and weights."""
    rng = np.random.default_rng(7)
    shapes = []
    for _ in range(case["graphs"]):
        n = int(rng.integers(max(60, case["n"] // 12), case["n"] + 1))
        degree = float(rng.uniform(5.0, 2.0 * case["degree"]))
        kind = str(rng.choice(["int", "lognormal", "unit"], p=[0.45, 0.45, 0.10]))
        shapes.append((n, min(degree, n / 6), kind))
    return shapes


def _graphs(case, seed):
    if case["kind"] == "batch":
        return [(n, *_csr(n, d, case["scale"], k, case["sigma"], 1000 * seed + i)) for i, (n, d, k) in enumerate(_batch_shapes(case))]
    return [(case["n"], *_csr(case["n"], case["degree"], case["scale"], case["weights"], case["sigma"], seed))]


def _pick_sources(case, order, seed):
    """A contiguous block of the all-sources order, as a program that splits an all-sources job takes it."""
    k = case["sources"]
    at = int(np.random.default_rng(seed).integers(0, max(1, len(order) - k + 1)))
    return np.ascontiguousarray(order[at:at + k])


def prepare(case, seed):
    kind = case["kind"]
    graphs = _graphs(case, seed)
    if kind == "batch":
        return {"case": case, "batch": Batch(graphs), "graphs": graphs}
    n, row_ptr, col, w = graphs[0]
    if kind == "train":
        weight = torch.tensor(w, device=_device(), requires_grad=True)
        return {"case": case, "n": n, "row_ptr": row_ptr, "col": col, "w": weight}
    state = {"case": case, "graph": Graph(n, row_ptr, col, w), "w": w, "sources": None}
    if kind == "rows":
        state["sources"] = np.random.default_rng(seed).choice(n, case["sources"], replace=False)
    elif kind != "scc" and case["sources"] > 0:
        # the million-vertex graph is sampled uniformly, the others by blocks of the locality order
        order = np.random.default_rng(seed).permutation(n) if n > 500000 else state["graph"].source_order()
        state["sources"] = _pick_sources(case, order, seed)
    return state


_PER = ("sum", "max", "sum_inv")


def _summary(r):
    out = {"means": np.array([r.cpl, r.efficiency, r.diameter], np.float64),
           "counts": np.array([r.unreachable, r.reached_pairs, r.traversed_arcs, r.hist_overflow], np.int64)}
    if r.hist is not None:
        out["hist"] = r.hist.astype(np.int64)
    if r.per_source is not None:
        for k in _PER:
            out[k] = r.per_source[k]
        out["unreachable"] = r.per_source["unreachable"].astype(np.int64)
    return out


def run(state):
    case = state["case"]
    kind, hist = case["kind"], case["hist"]
    if kind == "batch":
        # a cohort's histograms share one range
        results, bc = state["batch"].run("brandes", hist_bins=hist, hist_max=60.0 if hist else 0.0, per_source=True, use_cuda_graph=True)
        parts = [_summary(r) for r in results]
        out = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
        out["bc"] = np.concatenate(bc)
        return out
    if kind == "train":
        w = state["w"]
        w.grad = None
        metrics = apsp_metrics(w, state["n"], state["row_ptr"], state["col"])
        (metrics[0] - metrics[1]).backward()
        return {"metrics": metrics.detach(), "grad": w.grad}
    g, sources = state["graph"], state["sources"]
    if kind == "apsp":
        return _summary(g.apsp(sources, hist_bins=hist, per_source=True))
    if kind == "apsp_inverse":
        return _summary(g.apsp(sources, metric="inverse", hist_bins=hist, per_source=True))
    if kind == "rows":
        return {"rows": g.sssp_rows(sources)}
    if kind == "brandes":
        bc, r = g.brandes(sources, hist_bins=hist, per_source=True)
        return {"bc": bc, **_summary(r)}
    if kind == "grad":
        g.update_weights(state["w"])
        dcpl, deff, r = g.apsp_grad(sources)
        return {"dcpl": dcpl, "deff": deff, **_summary(r)}
    if kind == "scc":
        r = g.scc()
        return {"counts": np.array([r["number_components"], r["largest_component_size"]], np.int64), "component": r["component"]}
    raise ValueError(kind)


def work(case):
    """Bytes: each arc (target and weight) and row offset once, each output once. Flops: an addition and a comparison
    per (source, arc), the relaxation of a shortest-path search, and as much again for each of sigma and delta."""
    shapes = [(n, n * d, n) for n, d, _ in _batch_shapes(case)] if case["kind"] == "batch" else \
        [(case["n"], case["n"] * case["degree"], case["sources"] or case["n"])]
    kind = case["kind"]
    moved = flops = 0.0
    for n, m, s in shapes:
        moved += 12.0 * m + 8.0 * n
        if kind == "scc":
            moved += 4.0 * n
            continue
        flops += 2.0 * m * s * (3.0 if kind in ("brandes", "grad", "train", "batch") else 1.0)
        moved += 8.0 * s * n if kind == "rows" else 36.0 * s
        moved += 8.0 * n if kind in ("brandes", "batch") else 16.0 * m if kind in ("grad", "train") else 0.0
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------------------------------------- 64-bit reference
def _reference(n, row_ptr, col, length, sources, want):
    """Distances by Bellman-Ford rounds, path counts and dependencies by rounds over the shortest-path DAG, in float64
    torch; sums in extended precision. want: "rows", "apsp", "brandes" or "grad"."""
    dev = _device()
    src = torch.as_tensor(np.repeat(np.arange(n), np.diff(row_ptr)), device=dev)
    dst = torch.as_tensor(col.astype(np.int64), device=dev)
    ln = torch.as_tensor(length, device=dev)
    m = int(src.numel())
    out = {"rows": [], "sum": [], "max": [], "sum_inv": [], "bc": torch.zeros(n, dtype=torch.float64, device=dev),
           "c": torch.zeros(m, dtype=torch.float64, device=dev), "cg": torch.zeros(m, dtype=torch.float64, device=dev), "reached": 0}
    width = max(1, min(32, int(2.0e8 / max(m, 1))))
    for at in range(0, len(sources), width):
        s = torch.as_tensor(np.asarray(sources[at:at + width], dtype=np.int64), device=dev)
        k = int(s.numel())
        lanes = torch.arange(k, device=dev)
        d = torch.full((n, k), math.inf, dtype=torch.float64, device=dev)
        d[s, lanes] = 0.0
        while m:
            new = d.scatter_reduce(0, dst[:, None].expand(-1, k), d[src] + ln[:, None], "amin")
            if torch.equal(new, d):
                break
            d = new
        rows = d.t().cpu().numpy()
        if want == "rows":
            out["rows"].append(rows)
            continue
        fin = np.isfinite(rows)
        ext = np.where(fin, rows, 0.0).astype(np.longdouble)
        with np.errstate(divide="ignore"):
            inv = np.where(fin & (rows > 0), 1.0 / rows, 0.0).astype(np.longdouble)
        out["sum"].append(ext.sum(1))
        out["sum_inv"].append(inv.sum(1))
        out["max"].append(np.where(fin, rows, 0.0).max(1))
        out["reached"] += int(fin.sum()) - k
        if want == "apsp":
            continue
        dag = (d[src] + ln[:, None] == d[dst]) & torch.isfinite(d[dst])
        dag[(dst[:, None] == s[None, :])] = False
        e, lane = torch.nonzero(dag, as_tuple=True)
        del dag
        u, x = src[e] * k + lane, dst[e] * k + lane
        sigma = torch.zeros(n * k, dtype=torch.float64, device=dev)
        start = sigma.clone()
        start[s * k + lanes] = 1.0
        sigma = start
        depth = 0  # rounds until the counts (integers) stand: the longest shortest path, in arcs
        while True:
            new = start.index_add(0, x, sigma[u])
            if torch.equal(new, sigma):
                break
            sigma, depth = new, depth + 1
        share = sigma[u] / sigma[x]
        delta = torch.zeros(n * k, dtype=torch.float64, device=dev)
        dg = torch.zeros_like(delta)
        g = torch.where(d > 0, 1.0 / (d * d), torch.zeros_like(d)).reshape(-1)
        for _ in range(depth):
            if want == "grad":
                dg = torch.zeros_like(dg).index_add_(0, u, share * (g[x] + dg[x]))
            delta = torch.zeros_like(delta).index_add_(0, u, share * (1.0 + delta[x]))
        if want == "grad":
            out["c"].index_add_(0, e, share * (1.0 + delta[x]))
            out["cg"].index_add_(0, e, share * (g[x] + dg[x]))
        delta[s * k + lanes] = 0.0
        out["bc"] += delta.reshape(n, k).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "scc" or (case["sources"] > 0 and kind != "rows"):
        return None  # whole numbers; sources taken from the library's own order
    shapes = [(n, n * d, n) for n, d, _ in _batch_shapes(case)] if kind == "batch" else [(case["n"], case["n"] * case["degree"], case["sources"] or case["n"])]
    # rounds x passes over (arc, source) pairs: about 20 seconds at the most
    if sum(m * s for _, m, s in shapes) > (4.0e9 if kind in ("apsp", "apsp_inverse", "rows") else 1.0e9) or max(n for n, _, _ in shapes) > 200000:
        return None
    parts = []
    for n, row_ptr, col, w in _graphs(case, seed):
        sources = np.random.default_rng(seed).choice(n, case["sources"], replace=False) if kind == "rows" else np.arange(n)
        want = {"rows": "rows", "apsp": "apsp", "apsp_inverse": "apsp", "brandes": "brandes", "batch": "brandes"}.get(kind, "grad")
        r = _reference(n, row_ptr, col, 1.0 / w if kind == "apsp_inverse" else w, sources, want)
        if want == "rows":
            return {"rows": np.concatenate(r["rows"])}
        total = [np.concatenate(r[k]) for k in _PER]
        reached = np.longdouble(r["reached"])
        with np.errstate(divide="ignore", invalid="ignore"):
            cpl, eff = total[0].sum() / reached, total[2].sum() / reached
        scalars = np.array([cpl, eff, total[1].max()], np.float64)
        if kind == "train":
            return {"metrics": scalars[:2], "grad": (r["c"] / r["reached"] + r["cg"] / r["reached"]).cpu().numpy()}
        part = {"means": scalars, "sum": total[0].astype(np.float64), "max": total[1].astype(np.float64), "sum_inv": total[2].astype(np.float64)}
        if want == "brandes":
            part["bc"] = r["bc"].cpu().numpy()
        if want == "grad":
            part["dcpl"] = (r["c"] / r["reached"]).cpu().numpy()
            part["deff"] = (-r["cg"] / r["reached"]).cpu().numpy()
            for k in _PER:  # the gradient's public call returns no per-source arrays
                part.pop(k)
        parts.append(part)
    return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
