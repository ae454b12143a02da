"""Timed workloads of the KODAMA.matrix hot path through its public entry points.

Every case is one call a user's program makes, on seeded synthetic data of the
kinds in kodama_gb300.datasets.  ``listed()`` gives the fixed workloads,
``draw(rng)`` further ones of the same ranges; ``prepare`` makes the inputs,
``run`` makes the call and returns its whole outputs, ``work`` counts the bytes
and operations the result cannot do without, and ``exact`` restates the cases
whose outputs are computed numbers in 64 bits with plain torch.

Host arrays go in as numpy, as from R or a file; ``resident`` cases keep the
data matrix and the label matrix on the device, as a program does that goes on
working there.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import kodama_gb300 as kg
from kodama_gb300 import datasets

SEED = 1234  # the call's own seed, as in the reference's defaults and the benchmark


def listed():
    return [
        # the smallest work a user sees: correcting the graph of a 1000-row data set (three launches)
        dict(name="proximity_1k", kind="proximity", n=1000, K=50, runs=20),
        # the same step at the benchmark's size: 20000 rows, 100 runs
        dict(name="proximity_20k", kind="proximity", n=20000, K=30, runs=100),
        # the exact neighbour graph alone, at the default number of neighbours and an odd row count
        dict(name="graph_default_20k", kind="graph", n=20011, d=50, K=100, metric="euclidean"),
        # the exact graph under the cosine metric (spectra, embeddings: wider rows)
        dict(name="graph_cosine_12k", kind="graph", n=12000, d=100, K=30, metric="cosine"),
        # cross-validated kNN accuracy of a labelled data set, R's defaults (cosine, k = 10, 10 folds)
        dict(name="knncv_10k", kind="knncv", n=10000, d=50, k=10, folds=10, metric="cosine"),
        # one label evolution on raw data, the defaults of CoreKNN (100 cycles, k = 30, 10 folds)
        dict(name="core_knn_5k", kind="core_knn", n=5003, d=40, k=30, cycles=100, folds=10, classes=50,
             metric="euclidean"),
        # one label evolution with PLS-LDA as the predictor, stratified folds as in R
        dict(name="core_plslda_2k", kind="core_plslda", n=2001, d=50, components=5, cycles=30, folds=10, classes=20),
        # KODAMA.matrix on a small data set (three spirals): launches and latency
        dict(name="matrix_spirals_1k", kind="matrix", data="spirals", classifier="knn", n=1000, d=10, runs=20,
             cycles=20, K=50, knn_k=10, folds=10, splitting=0, components=5, metric="euclidean", resident=False),
        # KODAMA.matrix with every option at its default, on a mid-sized matrix of odd sizes
        dict(name="matrix_defaults_5k", kind="matrix", data="mixture", classifier="knn", n=4999, d=37, runs=100,
             cycles=20, K=100, knn_k=30, folds=5, splitting=0, components=50, metric="euclidean", resident=False),
        # the headline workload of the benchmark, data and labels resident in HBM
        dict(name="matrix_mixture_20k", kind="matrix", data="mixture", classifier="knn", n=20000, d=50, runs=100,
             cycles=100, K=30, knn_k=30, folds=10, splitting=50, components=50, metric="euclidean", resident=True),
        # the largest: 100000 rows with a decaying spectrum, default landmarks and splitting, from host memory
        dict(name="matrix_pca_100k", kind="matrix", data="pca", classifier="knn", n=100000, d=50, runs=100,
             cycles=100, K=30, knn_k=30, folds=10, splitting=0, components=50, metric="euclidean", resident=False),
        # KODAMA.matrix with the PLS-LDA classifier on wide rows, the benchmark's configuration
        dict(name="matrix_pls_10k", kind="matrix", data="low_rank", classifier="pls", n=10000, d=200, runs=50,
             cycles=50, K=30, knn_k=30, folds=10, splitting=0, components=5, metric="euclidean", resident=False),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over [lo, hi] by its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["proximity", "graph", "knncv", "core_knn", "core_plslda", "matrix", "matrix", "matrix_pls"])
    if kind == "proximity":
        return dict(kind=kind, n=_log_int(rng, 500, 30000), K=_log_int(rng, 10, 100), runs=_log_int(rng, 10, 130))
    if kind == "graph":
        return dict(kind=kind, n=_log_int(rng, 800, 30000), d=_log_int(rng, 8, 128), K=_log_int(rng, 10, 100),
                    metric=rng.choice(["euclidean", "euclidean", "cosine", "inner_product"]))
    if kind == "knncv":
        return dict(kind=kind, n=_log_int(rng, 500, 15000), d=_log_int(rng, 8, 100), k=rng.randint(3, 30),
                    folds=rng.choice([5, 10]), metric=rng.choice(["cosine", "cosine", "euclidean", "inner_product"]))
    if kind == "core_knn":
        return dict(kind=kind, n=_log_int(rng, 500, 10000), d=_log_int(rng, 8, 100), k=rng.randint(5, 30),
                    cycles=rng.randint(20, 100), folds=rng.choice([5, 10]), classes=rng.randint(10, 100),
                    metric=rng.choice(["euclidean", "euclidean", "cosine"]))
    if kind == "core_plslda":
        return dict(kind=kind, n=_log_int(rng, 300, 4000), d=_log_int(rng, 8, 100), components=rng.randint(2, 8),
                    cycles=rng.randint(10, 30), folds=rng.choice([5, 10]), classes=rng.randint(5, 40))
    if kind == "matrix":
        # wider graphs, wider rows and the other metrics up to 20000 rows; above, the benchmark's kind
        n = _log_int(rng, 500, 100000)
        big = n > 20000
        return dict(kind="matrix", data=rng.choice(["mixture", "mixture", "pca"]), classifier="knn", n=n,
                    d=_log_int(rng, 8, 50 if big else 100), runs=_log_int(rng, 10, 100),
                    cycles=rng.randint(10, 100), K=30 if big else rng.choice([30, 50, 100]),
                    knn_k=rng.randint(5, 30), folds=rng.choice([5, 10]), splitting=rng.choice([0, 50, 100]),
                    components=50, resident=rng.random() < 0.5,
                    metric="euclidean" if big else rng.choice(["euclidean", "euclidean", "euclidean", "cosine"]))
    return dict(kind="matrix", data=rng.choice(["mixture", "low_rank"]), classifier="pls",
                n=_log_int(rng, 500, 8000), d=_log_int(rng, 10, 150), runs=_log_int(rng, 10, 50),
                cycles=rng.randint(10, 50), K=rng.choice([30, 50]), knn_k=rng.randint(5, 30),
                folds=rng.choice([5, 10]), splitting=0, components=rng.randint(2, 5), metric="euclidean",
                resident=rng.random() < 0.5)


def _data(kind, n, d, seed):
    if kind == "spirals":
        x, y = datasets.spirals(n=n, seed=seed)
    elif kind == "low_rank":
        x, y = datasets.low_rank(n=n, d=d, seed=seed)
    elif kind == "pca":
        x, y = datasets.pca_mixture(n=n, d=d, seed=seed)
    else:
        x, y = datasets.gaussian_mixture(n=n, d=d, seed=seed)
    return np.ascontiguousarray(x, np.float32), np.ascontiguousarray(y, np.int32)


def _start_labels(x, classes, seed):
    """The rows' nearest of `classes` random rows, labelled 1..classes: the kind of start an evolution gets."""
    rng = np.random.default_rng(seed + 77)
    c = x[rng.choice(len(x), classes, replace=False)]
    d2 = (c * c).sum(1)[None, :] - 2.0 * (x @ c.T)
    return (np.argmin(d2, axis=1) + 1).astype(np.int32)


def _proximity_inputs(case, seed):
    """A one-based graph whose neighbours mostly share the row's cluster, and run labels that mostly follow it."""
    n, K, runs = case["n"], case["K"], case["runs"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    cluster = torch.arange(n, device="cuda") * 12 // n
    first = (cluster * n + 11) // 12
    size = torch.clamp(((cluster + 1) * n + 11) // 12 - first, min=1)
    u = torch.rand(n, K, generator=g, device="cuda", dtype=torch.float64)
    inside = first[:, None] + (u * size[:, None]).long()
    anywhere = torch.randint(0, n, (n, K), generator=g, device="cuda")
    far = torch.rand(n, K, generator=g, device="cuda") < 0.1
    idx = torch.clamp(torch.where(far, anywhere, inside), max=n - 1)
    dist = torch.sort(torch.rand(n, K, generator=g, device="cuda") * 4.0 + 0.5, dim=1).values
    noise = torch.randint(1, 13, (runs, n), generator=g, device="cuda")
    keep = torch.rand(runs, n, generator=g, device="cuda") < 0.8
    labels = torch.where(keep, cluster[None, :] + 1, noise)
    return (idx + 1).to(torch.int32).contiguous(), dist.contiguous(), labels.to(torch.int32).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "proximity":
        idx, dist, labels = _proximity_inputs(case, seed)
        return dict(case=case, idx=idx, dist=dist, labels=labels)
    data = case.get("data", "low_rank" if "pls" in kind else "mixture")
    x, y = _data(data, case["n"], case["d"], seed)
    state = dict(case=case, x=x, y=y)
    if kind in ("core_knn", "core_plslda"):
        state["start"] = _start_labels(x, min(case["classes"], case["n"] // 4), seed)
    if kind == "matrix" and case["resident"]:
        state["x"] = torch.from_numpy(x).cuda()
        state["res"] = torch.empty((case["runs"], x.shape[0]), dtype=torch.int32, device="cuda")
    return state


def _core_outputs(r):
    return dict(clbest=r.clbest, cvpredbest=r.cvpredbest, folds=r.fold_assignments, acc=r.vect_acc,
                score=r.vect_score, proposal=r.proposal_size, active=r.active_classes, flags=r.flags,
                accbest=float(r.accbest), scorebest=float(r.scorebest), counters=r.counters)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "proximity":
        # the correction works in place: the caller keeps its raw graph
        idx, dist = state["idx"].clone(), state["dist"].clone()
        kg.KODAMADissimilarityInPlace_device(idx, dist, state["labels"])
        return idx, dist
    if kind == "graph":
        return kg.knn_graph(state["x"], case["K"], metric=case["metric"])
    if kind == "knncv":
        r = kg.KNNCV(state["x"], state["y"], folds=case["folds"], k=case["k"], metric=case["metric"], seed=SEED)
        return dict(pred=r.predicted_labels, folds=r.fold_assignments, acc=r.global_accuracy,
                    confusion=r.confusion.counts)
    if kind == "core_knn":
        r = kg.CoreKNN(state["x"], state["start"], cycles=case["cycles"], folds=case["folds"], k=case["k"],
                       metric=case["metric"], seed=SEED)
        return _core_outputs(r)
    if kind == "core_plslda":
        r = kg.CorePLSLDA(state["x"], state["start"], cycles=case["cycles"], folds=case["folds"],
                          max_components=case["components"], fixed_components=case["components"], seed=SEED,
                          cv_seed=SEED)
        return _core_outputs(r)
    r = kg.KODAMA_matrix(state["x"], runs=case["runs"], cycles=case["cycles"], splitting=case["splitting"],
                         graph_neighbors=case["K"], folds=case["folds"], knn_k=case["knn_k"], seed=SEED,
                         classifier=case["classifier"], components=case["components"], metric=case["metric"],
                         materialize_graph=True, res_out=state.get("res"))
    return dict(res=state["res"] if case["resident"] else r.res, acc=r.acc, trace=r.v,
                hashes=r.run_hashes.view(np.int64), counters=r.run_counters, cycles=r.cycle_diag,
                knn_idx=r.knn_idx, knn_dist=r.knn_dist, landmarks=r.effective_landmarks)


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "proximity":
        K, runs = case["K"], case["runs"]
        return {"bytes": 4 * runs * n + 2 * 8 * n * K, "flops": 2 * n * K * runs}
    d = case["d"]
    if kind == "graph":
        return {"bytes": 4 * n * d + 8 * n * case["K"], "flops": 3 * n * n * d}
    if kind == "knncv":
        return {"bytes": 4 * n * d + 12 * n, "flops": 3 * n * n * d}
    if kind == "core_knn":
        # the search, then one vote per row and cycle at most
        return {"bytes": 4 * n * d + 16 * n, "flops": 3 * n * n * d + (case["cycles"] + 1) * n * case["k"]}
    if kind == "core_plslda":
        # per fold and component: one pass over the training rows for the scores and one for the loadings
        return {"bytes": 4 * n * d + 16 * n, "flops": (case["cycles"] + 1) * (case["folds"] - 1) * 4 * n * d * case["components"]}
    M, T, K = case["runs"], case["cycles"], case["K"]
    L = min(10000, n - 1) if n > 10000 else int(math.ceil(0.75 * n))
    k = case["splitting"] or (100 if n < 40000 else 300)
    flops = 2 * n * n * d + 2 * 11 * k * d * (n + M * L)
    if case["classifier"] == "pls":
        flops += (T + 1) * M * (case["folds"] - 1) * 4 * L * d * case["components"]
    else:
        flops += (T + 1) * M * L * case["knn_k"]
    return {"bytes": 4 * n * d + 4 * M * n + 8 * n * K, "flops": flops}


def exact(case, seed):
    if case["kind"] == "graph":
        x = torch.from_numpy(_data("mixture", case["n"], case["d"], seed)[0]).cuda().double()
        n, K, metric = case["n"], case["K"], case["metric"]
        if metric == "cosine":
            x = x / x.norm(dim=1, keepdim=True)
        sq = (x * x).sum(1)
        out = torch.empty((n, K), dtype=torch.float64, device="cuda")
        for a in range(0, n, 2048):
            b = min(n, a + 2048)
            g = x[a:b] @ x.T
            v = sq[a:b, None] + sq[None, :] - 2.0 * g if metric == "euclidean" else -g
            v[torch.arange(b - a), torch.arange(a, b)] = math.inf
            v = torch.topk(v, K, dim=1, largest=False, sorted=True).values
            if metric == "euclidean":
                v = v.clamp(min=0.0).sqrt()
            else:
                v = 1.0 + v
                v = v.clamp(min=0.0) if metric == "cosine" else v
            out[a:b] = v
        return None, out
    if case["kind"] == "proximity":
        idx, dist, labels = _proximity_inputs(case, seed)
        n, K = idx.shape
        lab = labels.T.contiguous()
        out = torch.empty((n, K), dtype=torch.float64, device="cuda")
        for a in range(0, n, 2048):
            b = min(n, a + 2048)
            agree = (lab[a:b, None, :] == lab[idx[a:b].long() - 1]).double().mean(dim=2)
            v = (1.0 + dist[a:b].double()) / (agree * agree)
            out[a:b] = torch.sort(v, dim=1).values
        return None, out
    # the other calls return labels, and accuracies that are functions of them
    return None
