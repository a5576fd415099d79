"""Performance cases: the calls a user of this framework makes, over the range of sizes they make them at.

``listed()`` names twelve of them; ``draw(rng)`` gives others from the same
ranges.  A case is a plain dict; ``prepare`` makes its inputs on the GPU from a
seed, ``run`` makes one pass through the public entry points (``knn_arrays``,
``IVFFlatIndex.build``, ``ProbeModel.train`` and ``ivf_search_device`` of the
package, the ``mann_*_device`` calls of the C ABI), ``work`` counts what the
path cannot do without and ``exact`` computes the same outputs in 64 bits with
plain torch.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import manifoldann_gb300 as M
from manifoldann_gb300 import _lib

METRICS = {"euclidean": M.Euclidean, "sqeuclidean": M.SqEuclidean, "cosine": M.CosineDist}
METRIC_CODES = {"euclidean": _lib.METRIC_EUCLIDEAN, "sqeuclidean": _lib.METRIC_SQEUCLIDEAN,
                "cosine": _lib.METRIC_COSINE}
PRECISIONS = {"fp32": _lib.PREC_FP32, "bf16": _lib.PREC_BF16, "fp16": _lib.PREC_FP16, "auto": _lib.PREC_AUTO}


def listed():
    return [
        # one query against a small indexed set kept on the device, from host memory: the latency of the smallest call
        {"name": "query_one", "kind": "knn", "via": "handle", "data": "normal", "n": 10_000, "q": 1, "d": 64, "k": 10,
         "metric": "sqeuclidean", "precision": "fp32", "ties": False, "graph": False},
        # plain exact kNN, the default form: a batch of queries against a small set
        {"name": "plain_10k_64", "kind": "knn", "via": "device", "data": "normal", "n": 10_000, "q": 1_000, "d": 64,
         "k": 10, "metric": "sqeuclidean", "precision": "fp32", "ties": False, "graph": False},
        # build_knn_graph with its defaults (Euclidean distance, FP32 form) on a set of ragged size
        {"name": "graph_fp32_20k_100", "kind": "knn", "via": "device", "data": "aniso", "n": 20_011, "q": 20_011,
         "d": 100, "k": 15, "metric": "euclidean", "precision": "fp32", "ties": False, "graph": True},
        # held-out queries in the tensor-core form with the FP64 order of near-ties
        {"name": "queries_60k_784", "kind": "knn", "via": "device", "data": "quantized", "n": 60_000, "q": 10_000,
         "d": 784, "k": 10, "metric": "sqeuclidean", "precision": "bf16", "ties": True, "graph": False},
        # the whole self-kNN graph of the same set, the largest search
        {"name": "graph_60k_784", "kind": "knn", "via": "device", "data": "quantized", "n": 60_000, "q": 60_000,
         "d": 784, "k": 10, "metric": "sqeuclidean", "precision": "bf16", "ties": True, "graph": True},
        # angular search where the library picks the form
        {"name": "cosine_290k_256", "kind": "knn", "via": "device", "data": "angular", "n": 290_000, "q": 10_000,
         "d": 256, "k": 20, "metric": "cosine", "precision": "auto", "ties": False, "graph": False},
        # graphs of many point clouds of uneven size in one call, as build_knn_graphs makes it (FP32 form)
        {"name": "clouds_fp32", "kind": "clouds", "sets": 24, "lo": 2_000, "hi": 50_000, "d": 32, "k": 15,
         "metric": "sqeuclidean", "precision": "fp32"},
        # the same call in the tensor-core form
        {"name": "clouds_bf16", "kind": "clouds", "sets": 24, "lo": 2_000, "hi": 50_000, "d": 32, "k": 15,
         "metric": "sqeuclidean", "precision": "bf16"},
        # the weighted graph's second half: every node's tangent space, then every edge's weight
        {"name": "geometry_32", "kind": "geometry", "sets": 16, "lo": 2_000, "hi": 30_000, "d": 32, "k": 15, "dim": 2,
         "rule": 4},
        # serving: a batch of queries routed to the lists of an inverted-file index and scanned there
        {"name": "ivf_search_1m_128", "kind": "ivf_search", "n": 1_000_000, "q": 10_000, "d": 128, "nlist": 4_096,
         "nprobe": 4, "k": 10},
        # building that kind of index from host data: k-means++, Lloyd, the lists
        {"name": "ivf_build_262k_128", "kind": "ivf_build", "n": 262_144, "d": 128, "nlist": 1_024, "iters": 25},
        # training the learned routing: forward, backward and AdamW over shuffled batches
        {"name": "probe_train_128", "kind": "probe_train", "nq": 65_536, "din": 128, "hidden": 512, "nout": 4_096,
         "labels": 10, "batch": 1_024, "epochs": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; sizes are spread over their logarithm."""
    kind = rng.choice(["one", "plain", "graph32", "tensor", "tensor_graph", "clouds", "geometry", "ivf_search",
                       "ivf_build", "probe_train"])
    if kind == "one":  # a few host queries against a device-resident set
        return {"kind": "knn", "via": "handle", "data": "normal", "n": _log(rng, 1_000, 60_000),
                "q": rng.choice([1, 1, 2, 3, 7, 17]), "d": _log(rng, 16, 784), "k": rng.choice([1, 5, 10, 20]),
                "metric": rng.choice(list(METRICS)), "precision": "fp32", "ties": False, "graph": False}
    if kind == "plain":
        return {"kind": "knn", "via": "device", "data": rng.choice(["normal", "aniso"]), "n": _log(rng, 2_000, 60_000),
                "q": _log(rng, 33, 10_000), "d": _log(rng, 8, 256), "k": rng.choice([1, 5, 10, 20, 33]),
                "metric": rng.choice(list(METRICS)), "precision": "fp32", "ties": rng.random() < 0.25, "graph": False}
    if kind == "graph32":
        n = _log(rng, 2_000, 30_000)
        return {"kind": "knn", "via": "device", "data": rng.choice(["normal", "aniso"]), "n": n, "q": n,
                "d": _log(rng, 8, 200), "k": rng.choice([5, 10, 15, 20]),
                "metric": rng.choice(["euclidean", "sqeuclidean"]), "precision": "fp32", "ties": False, "graph": True}
    if kind == "tensor":
        return {"kind": "knn", "via": "device", "data": rng.choice(["quantized", "angular", "aniso"]),
                "n": _log(rng, 8_000, 290_000), "q": _log(rng, 100, 10_000), "d": _log(rng, 128, 800),
                "k": rng.choice([1, 10, 20]), "metric": rng.choice(list(METRICS)),
                "precision": rng.choice(["bf16", "auto", "auto"]), "ties": rng.random() < 0.5, "graph": False}
    if kind == "tensor_graph":
        n = _log(rng, 8_000, 60_000)
        return {"kind": "knn", "via": "device", "data": rng.choice(["quantized", "aniso"]), "n": n, "q": n,
                "d": _log(rng, 128, 784), "k": rng.choice([5, 10, 20]),
                "metric": rng.choice(["euclidean", "sqeuclidean"]), "precision": rng.choice(["bf16", "auto"]),
                "ties": rng.random() < 0.5, "graph": True}
    if kind == "clouds":
        lo = _log(rng, 500, 5_000)
        return {"kind": "clouds", "sets": rng.randint(4, 24), "lo": lo, "hi": _log(rng, lo, 50_000),
                "d": rng.choice([3, 16, 30, 32, 48]), "k": rng.choice([5, 10, 15, 20]),
                "metric": rng.choice(["euclidean", "sqeuclidean"]), "precision": rng.choice(["fp32", "bf16"])}
    if kind == "geometry":
        return {"kind": "geometry", "sets": rng.randint(2, 16), "lo": 1_000, "hi": _log(rng, 2_000, 30_000),
                "d": rng.choice([3, 8, 20, 32, 50]), "k": rng.randint(8, 30), "dim": rng.choice([0, 1, 2, 3]),
                "rule": rng.randint(0, 4)}
    if kind == "ivf_search":
        n = _log(rng, 50_000, 1_000_000)
        return {"kind": "ivf_search", "n": n, "q": _log(rng, 100, 10_000), "d": rng.choice([64, 96, 100, 128]),
                "nlist": max(64, min(4_096, n // rng.randint(200, 600))), "nprobe": rng.randint(1, 12),
                "k": rng.choice([1, 10, 20])}
    if kind == "ivf_build":
        return {"kind": "ivf_build", "n": _log(rng, 20_000, 262_144), "d": rng.choice([48, 64, 100, 128]),
                "nlist": _log(rng, 64, 1_024), "iters": rng.randint(5, 25)}
    return {"kind": "probe_train", "nq": _log(rng, 4_000, 65_536), "din": rng.choice([64, 96, 128]),
            "hidden": rng.choice([128, 256, 512]), "nout": _log(rng, 256, 4_096), "labels": 10,
            "batch": rng.choice([512, 1_024]), "epochs": rng.randint(1, 2)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)


def _points(data, n, d, g):
    """n rows of d floats on the GPU in the distributions of ``synthetic``; mixtures also give the component ids."""
    kw = {"device": "cuda", "generator": g}
    if data == "normal":
        return torch.randn((n, d), **kw), None
    if data == "quantized":
        centres = torch.rand((10, d), **kw) * 0.8 + 0.1
        comp = torch.randint(0, 10, (n,), **kw)
        x = torch.randn((n, d), **kw).mul_(0.15).add_(centres[comp]).clamp_(0.0, 1.0)
        return x.mul_(255.0).round_().div_(255.0), comp
    if data == "angular":
        centres = torch.nn.functional.normalize(torch.randn((100, d), **kw), dim=1)
        comp = torch.randint(0, 100, (n,), **kw)
        x = torch.randn((n, d), **kw).mul_(0.3).add_(centres[comp])
        return x.div_(x.norm(dim=1, keepdim=True)), comp
    centres = torch.randn((1024, d), **kw)
    sig = torch.exp(torch.rand((1024, d), **kw) * math.log(10.0) + math.log(0.05))
    comp = torch.randint(0, 1024, (n,), **kw)
    return torch.randn((n, d), **kw).mul_(sig[comp]).add_(centres[comp]), comp


def _knn_inputs(case, seed):
    g = _gen(seed)
    n, q = case["n"], 0 if case["graph"] else case["q"]
    x, _ = _points(case["data"], n + q, case["d"], g)
    return x[:n], (x[:n] if case["graph"] else x[n:].contiguous())


def _cloud_sizes(case):
    """Sizes log-uniform in [lo, hi], the same for every seed."""
    r = random.Random(case["sets"] * 1_000_003 + case["lo"] * 101 + case["hi"])
    return [_log(r, case["lo"], case["hi"]) for _ in range(case["sets"])]


def _clouds(case, seed):
    """Swiss rolls, spheres and tori in R^3, rotated into R^d, with noise; back to back."""
    g, d = _gen(seed), case["d"]
    kw = {"device": "cuda", "generator": g}
    rot = torch.linalg.qr(torch.randn((d, d), generator=torch.Generator().manual_seed(int(seed))))[0].cuda()
    sizes = _cloud_sizes(case)
    out = []
    for i, n in enumerate(sizes):
        u, v = torch.rand((n,), **kw), torch.rand((n,), **kw)
        if i % 3 == 0:
            t = 1.5 * math.pi * (1 + 2 * u)
            p = torch.stack([t * torch.cos(t), 21 * v, t * torch.sin(t)], 1) / 10.0
        elif i % 3 == 1:
            p = torch.nn.functional.normalize(torch.randn((n, 3), **kw), dim=1)
        else:
            th, ph = 2 * math.pi * u, 2 * math.pi * v
            rr = 1.0 + 0.35 * torch.cos(th)
            p = torch.stack([rr * torch.cos(ph), rr * torch.sin(ph), 0.35 * torch.sin(th)], 1)
        # three products in a fixed order: the same bits on every run
        x = p[:, 0:1] * rot[0] + p[:, 1:2] * rot[min(1, d - 1)] + p[:, 2:3] * rot[min(2, d - 1)]
        out.append(x + 0.01 * torch.randn((n, d), **kw))
    offs = np.zeros(len(sizes) + 1, np.int64)
    offs[1:] = np.cumsum(sizes)
    return torch.cat(out).contiguous(), offs


def _smallest(x, y, k, metric="sqeuclidean", drop_self=False, want_ids=False, dtype=torch.float64, step=2048):
    """The k smallest distances of every row of y to the rows of x, ascending, a block of rows at a time."""
    xb = x.to(dtype)
    norms = (xb * xb).sum(1)
    vals, ids = [], []
    for s in range(0, y.shape[0], step):
        yb = y[s:s + step].to(dtype)
        dot = yb @ xb.T
        yn = (yb * yb).sum(1, keepdim=True)
        if metric == "cosine":
            v = (1.0 - dot / (yn.sqrt() * norms.sqrt())).clamp_(min=0.0)
        else:
            v = dot.mul_(-2.0).add_(norms).add_(yn).clamp_(min=0.0)
        if drop_self:
            r = torch.arange(yb.shape[0], device=v.device)
            v[r, r + s] = float("inf")
        kk = min(k, v.shape[1])
        w, i = torch.topk(v, kk, dim=1, largest=False, sorted=True)
        vals.append(w.sqrt() if metric == "euclidean" else w)
        if want_ids:
            ids.append(i)
    return (torch.cat(vals), torch.cat(ids)) if want_ids else torch.cat(vals)


def _neighbours(X, offs, k):
    """Global neighbour ids [N][k] of every point within its own cloud."""
    out = []
    for a, b in zip(offs[:-1], offs[1:]):
        _, i = _smallest(X[a:b], X[a:b], k, drop_self=True, want_ids=True)
        out.append(i + int(a))
    return torch.cat(out).to(torch.int32).contiguous()


def _inverted_file(case, seed):
    """Points, queries and an inverted file over them: centroids taken evenly over the mixture's components."""
    g = _gen(seed)
    n, q, nlist = case["n"], case["q"], case["nlist"]
    x, comp = _points("aniso", n + q, case["d"], g)
    X, Q = x[:n].contiguous(), x[n:].contiguous()
    order = torch.argsort(comp[:n], stable=True)
    at = torch.linspace(0, n - 1, nlist, device="cuda", dtype=torch.float64).round().long()
    cent = X[order[at]].contiguous()
    cn = (cent * cent).sum(1)
    assign = torch.cat([(cn - 2.0 * (X[s:s + 65536] @ cent.T)).argmin(1) for s in range(0, n, 65536)])
    ids = torch.argsort(assign, stable=True)
    offs = torch.zeros(nlist + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(torch.bincount(assign, minlength=nlist), 0)
    return X, Q, cent, offs, ids.to(torch.int32).contiguous()


def _probe_inputs(case, seed):
    """Training queries around the lists' centroids, the lists they should find, and starting parameters."""
    g = _gen(seed)
    kw = {"device": "cuda", "generator": g}
    nq, din, h, nout = case["nq"], case["din"], case["hidden"], case["nout"]
    cent = torch.randn((nout, din), **kw)
    own = torch.randint(0, nout, (nq, 1), **kw)
    other = torch.randint(0, nout, (nq, case["labels"]), **kw)
    labels = torch.where(torch.rand((nq, case["labels"]), **kw) < 0.7, own, other)
    queries = cent[own[:, 0]] + 0.3 * torch.randn((nq, din), **kw)
    parts = []
    for rows, cols in ((h, din), (h, h), (nout, h)):
        parts += [((torch.rand((rows * cols,), **kw) * 2 - 1) / math.sqrt(cols)),
                  ((torch.rand((rows,), **kw) * 2 - 1) / math.sqrt(cols))]
    parts.append(torch.zeros(1, device="cuda"))
    return (queries.cpu().numpy(), labels.to(torch.int32).cpu().numpy(),
            np.ascontiguousarray(torch.cat(parts).cpu().numpy()))


# ---------------------------------------------------------------- state
def prepare(case, seed):
    s = {"case": case, "lib": _lib.load()}
    kind = case["kind"]
    if kind == "knn":
        x, y = _knn_inputs(case, seed)
        if case["via"] == "handle":
            host = x.cpu().numpy().T  # d x n, points as columns
            s["index"] = M.build_index(M.BruteForceIndex, host, distance=METRICS[case["metric"]]())
            s["points"] = M.DeviceDataset(host)
            queries = y.cpu().numpy().T
            s["queries"] = np.ascontiguousarray(queries[:, 0]) if case["q"] == 1 else queries
        else:
            s["x"], s["y"] = x, y
            s["params"] = _lib.params(METRIC_CODES[case["metric"]], case["k"], PRECISIONS[case["precision"]], 0,
                                      _lib.FLAG_FP64_TIES if case["ties"] else 0)
            _outputs(s, y.shape[0], case["k"])
    elif kind == "clouds":
        s["x"], s["offs"] = _clouds(case, seed)
        s["params"] = _lib.params(METRIC_CODES[case["metric"]], case["k"], PRECISIONS[case["precision"]])
        _outputs(s, s["x"].shape[0], case["k"])
    elif kind == "geometry":
        s["x"], offs = _clouds(case, seed)
        s["nbrs"] = _neighbours(s["x"], offs, case["k"])
        N, maxd = s["x"].shape[0], case["dim"] or min(case["d"], case["k"])
        s["centres"] = torch.arange(N, dtype=torch.int32, device="cuda")
        s["pca"] = _lib.PcaParams(case["dim"], 0, 0.95)
        s["maxd"] = maxd
        s["dims"] = torch.empty(N, dtype=torch.int32, device="cuda")
        s["eig"] = torch.empty((N, maxd), device="cuda")
        s["basis"] = torch.empty((N, maxd, case["d"]), device="cuda")
        s["weights"] = torch.empty((N, case["k"]), device="cuda")
    elif kind == "ivf_search":
        s["x"], s["y"], s["cent"], s["offs"], s["lids"] = _inverted_file(case, seed)
        cent = s["cent"].cpu().numpy()
        s["index"] = M.IVFFlatIndex(np.asfortranarray(cent.T), (cent.astype(np.float64) ** 2).sum(1).astype(np.float32),
                                    s["offs"].cpu().numpy(), s["lids"].cpu().numpy(), case["d"], case["nprobe"],
                                    M.SqEuclidean(), M.Euclidean())
        _outputs(s, case["q"], case["k"])
    elif kind == "ivf_build":
        x, _ = _points("aniso", case["n"], case["d"], _gen(seed))
        s["host"], s["seed"] = x.cpu().numpy().T, int(seed)
    else:
        s["queries"], s["labels"], s["start"] = _probe_inputs(case, seed)
    torch.cuda.synchronize()
    return s


def _outputs(s, rows, k):
    s["ids"] = torch.empty((rows, k), dtype=torch.int32, device="cuda")
    s["dists"] = torch.empty((rows, k), dtype=torch.float32, device="cuda")


# ---------------------------------------------------------------- one pass
def run(s):
    case, lib = s["case"], s["lib"]
    kind = case["kind"]
    if kind == "knn" and case["via"] == "handle":
        return M.knn_arrays(s["index"], s["points"], s["queries"], case["k"], precision=case["precision"],
                            fp64_ties=case["ties"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "knn":
        x, y = s["x"], s["y"]
        if case["graph"]:
            _lib.check(lib.mann_knn_graph_device(s["params"], x.data_ptr(), x.shape[0], x.shape[1], 0,
                                                 s["ids"].data_ptr(), s["dists"].data_ptr(), None, stream))
        else:
            _lib.check(lib.mann_knn_device(s["params"], x.data_ptr(), x.shape[0], y.data_ptr(), y.shape[0], x.shape[1],
                                           s["ids"].data_ptr(), s["dists"].data_ptr(), None, stream))
        return s["ids"], s["dists"]
    if kind == "clouds":
        _lib.check(lib.mann_knn_graph_batched_device(s["params"], s["x"].data_ptr(), s["offs"].ctypes.data,
                                                     case["sets"], case["d"], 0, s["ids"].data_ptr(),
                                                     s["dists"].data_ptr(), None, stream))
        return s["ids"], s["dists"]
    if kind == "geometry":
        x, N = s["x"], s["x"].shape[0]
        _lib.check(lib.mann_local_pca_device(s["pca"], x.data_ptr(), N, case["d"], s["centres"].data_ptr(), None, N,
                                             s["nbrs"].data_ptr(), case["k"], s["maxd"], s["dims"].data_ptr(),
                                             s["eig"].data_ptr(), s["basis"].data_ptr(), stream))
        negative = C.c_int64(0)
        _lib.check(lib.mann_edge_weights_device(case["rule"], x.data_ptr(), N, case["d"], s["nbrs"].data_ptr(),
                                                case["k"], s["dims"].data_ptr(), s["basis"].data_ptr(), s["maxd"],
                                                s["weights"].data_ptr(), C.byref(negative), stream))
        return s["dims"], s["eig"], s["basis"], s["weights"], negative.value
    if kind == "ivf_search":
        M.ivf_search_device(s["index"], s["x"], s["y"], case["k"], case["nprobe"], s["ids"], s["dists"], stream,
                            centroids_dev=s["cent"], offsets_dev=s["offs"], ids_dev=s["lids"])
        return s["ids"], s["dists"]
    if kind == "ivf_build":
        index = M.IVFFlatIndex.build(s["host"], nlist=case["nlist"], kmeans_max_iters=case["iters"],
                                     distance=M.SqEuclidean(), seed=s["seed"])
        return index.centroids, index.list_offsets, index.list_ids, index.kmeans_iters
    model = M.ProbeModel(case["din"], case["nout"], (case["hidden"], case["hidden"]), use_prior=False,
                         batch=case["batch"], seed=7, params=s["start"])
    loss = model.train(s["queries"], s["labels"], case["epochs"])
    return loss, model.params()


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "knn":
        n, q, d, k = case["n"], case["q"], case["d"], case["k"]
        rows = n if case["graph"] else n + q
        return {"bytes": 4 * rows * d + 8 * q * k, "flops": 2 * n * q * d}
    if kind == "clouds":
        sizes = _cloud_sizes(case)
        N = sum(sizes)
        return {"bytes": 4 * N * case["d"] + 8 * N * case["k"], "flops": 2 * case["d"] * sum(m * m for m in sizes)}
    if kind == "geometry":
        N, d, k = sum(_cloud_sizes(case)), case["d"], case["k"]
        maxd = case["dim"] or min(d, k)
        gram = 2 * d * k * k  # the smallest way to the spectrum: one Gram matrix of the k neighbours
        return {"bytes": 4 * N * (d + k + 2 + maxd + maxd * d + k), "flops": N * (gram + 2 * k * d * (1 + 2 * maxd))}
    if kind == "ivf_search":
        n, q, d = case["n"], case["q"], case["d"]
        seen = min(n, n * q * case["nprobe"] // case["nlist"])  # points of the lists that some query probes
        scanned = q * case["nprobe"] * n // case["nlist"]
        return {"bytes": 4 * d * (seen + q + case["nlist"]) + 4 * seen + 8 * q * case["k"],
                "flops": 2 * d * (q * case["nlist"] + scanned)}
    if kind == "ivf_build":
        n, d, k = case["n"], case["d"], case["nlist"]
        return {"bytes": 4 * n * d + 4 * k * d + 4 * n, "flops": 2 * n * k * d * (case["iters"] + 2)}
    din, h, nout = case["din"], case["hidden"], case["nout"]
    weights = din * h + h * h + h * nout
    params = weights + 2 * h + nout + 1
    return {"bytes": 4 * case["nq"] * (din + case["labels"]) + 8 * params,
            "flops": 6 * weights * case["nq"] * case["epochs"]}


# ---------------------------------------------------------------- the same outputs in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        x, y = _knn_inputs(case, seed)
        return [None, _smallest(x, y, case["k"], case["metric"], drop_self=case["graph"])]
    if kind == "clouds":
        X, offs = _clouds(case, seed)
        return [None, torch.cat([_smallest(X[a:b], X[a:b], case["k"], case["metric"], drop_self=True)
                                 for a, b in zip(offs[:-1], offs[1:])])]
    if kind == "geometry":
        return _exact_geometry(case, seed)
    if kind == "ivf_search":
        return _exact_search(case, seed)
    # the build's and the training's random draws are the library's own: nothing outside it has their results
    return None


def _exact_geometry(case, seed):
    X, offs = _clouds(case, seed)
    nbrs = _neighbours(X, offs, case["k"]).long()
    N, d, k, rule = X.shape[0], case["d"], case["k"], case["rule"]
    maxd = case["dim"] or min(d, k)
    X = X.double()
    eig = torch.zeros((N, maxd), dtype=torch.float64, device="cuda")
    basis = torch.zeros((N, maxd, d), dtype=torch.float64, device="cuda")
    take = min(d, k, maxd)
    for s in range(0, N, 4096):
        i = torch.arange(s, min(N, s + 4096), device="cuda")
        V = X[nbrs[i]] - X[i][:, None, :]
        lam, U = torch.linalg.eigh(V.transpose(1, 2) @ V)  # ascending, d x d
        lam, U = lam.flip(1).clamp(min=0.0), U.flip(2)
        if case["dim"]:
            keep = torch.arange(take, device="cuda").expand(len(i), take) < case["dim"]
        else:
            share = torch.cumsum(lam[:, :min(d, k)], 1) / lam.sum(1, keepdim=True)
            keep = torch.cat([torch.zeros_like(share[:, :1]), share[:, :-1]], 1) < 0.95
            keep = keep[:, :take]
        eig[i, :take] = torch.where(keep, lam[:, :take], 0.0)
        basis[i, :take] = torch.where(keep[:, :, None], U[:, :, :take].transpose(1, 2), 0.0)
    w = torch.empty((N, k), dtype=torch.float64, device="cuda")
    for s in range(0, N, 16384):
        i = torch.arange(s, min(N, s + 16384), device="cuda")
        j = nbrs[i]
        v = X[j] - X[i][:, None, :]
        e = v.norm(dim=2)
        own = torch.einsum("nkd,nmd->nkm", v, basis[i]).norm(dim=2)
        other = torch.einsum("nkd,nkmd->nkm", v, basis[j]).norm(dim=2)
        if rule == 4:
            raw = (8.0 * e - own - other) / 6.0
            w[i] = torch.where(raw < 0.0, e, raw)
        else:
            w[i] = (e, own, 0.5 * (own + other), torch.maximum(own, other))[rule]
    return [None, eig, None, w, None]


def _exact_search(case, seed):
    X, Q, cent, offs, lids = _inverted_file(case, seed)
    nprobe, k, q = min(case["nprobe"], case["nlist"]), case["k"], case["q"]
    _, probes = _smallest(cent, Q, nprobe, want_ids=True)
    best = torch.full((q, nprobe, k), float("inf"), dtype=torch.float64, device="cuda")
    flat = probes.reshape(-1)
    order = torch.argsort(flat, stable=True)
    bounds = np.concatenate([[0], np.cumsum(torch.bincount(flat, minlength=case["nlist"]).cpu().numpy())])
    host = offs.cpu().numpy()
    for c in range(case["nlist"]):
        a, b = int(host[c]), int(host[c + 1])
        pairs = order[int(bounds[c]):int(bounds[c + 1])]
        if a == b or pairs.numel() == 0:
            continue
        v = _smallest(X[lids[a:b].long()], Q[pairs // nprobe], k)
        best[pairs // nprobe, pairs % nprobe, :v.shape[1]] = v
    return [None, torch.sort(best.reshape(q, -1), dim=1)[0][:, :k].contiguous()]
