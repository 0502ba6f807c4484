"""The workloads that the front end's speed is judged on.

Every case goes through the package's public entry points (``ops``, ``topo``,
``persistence`` and the C-ABI binding ``capi``) on seeded synthetic clouds of
the kinds that ``turbotops_gb300.synth`` makes. ``listed()`` holds the named
ones, ``draw(rng)`` gives others of the same ranges:

  dense        distance matrix, enclosing radius and the dimension-0 stage of
               one full Rips cloud: 64 (the smallest batch cloud) to 12,000
               points, any metric
  knn          exact kNN lists, 1,000 to 100,000 points, 2 to 64 coordinates
  knn_graph    the same lists made into the symmetric kNN graph
  knn_front    host points in, kNN flag complex front end out (host buffers)
  radius       radius graph of a low-dimensional cloud
  mst          H0 of the complete graph (sorted spanning-tree weights)
  batch        many uneven full Rips clouds in one captured graph
  topo         one training step: topological loss, gradient of the points
  persistence  the whole call: front end and host reduction
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import turbotops_gb300 as tg
from turbotops_gb300 import capi, ops, synth, topo

_CTX = None


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(torch.cuda.current_device())
    return _CTX


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest cloud of the batched workload on its own: a caller that
        # runs tiny clouds one by one waits for launches and round trips
        {"name": "dense_circle64", "op": "dense", "cloud": "circle", "n": 64, "dim": 3, "metric": "l2", "maxdim": 1},
        # the tie-heavy full Rips cloud (integer lattice in R^4, L1): every
        # distance is shared by many pairs
        {"name": "dense_lattice3000", "op": "dense", "cloud": "lattice", "n": 3000, "dim": 4, "metric": "l1",
         "maxdim": 2},
        # a full Rips cloud near the size where its matrix leaves the L2 cache
        # and the edge list has tens of millions of entries
        {"name": "dense_gauss12000", "op": "dense", "cloud": "gauss", "n": 12000, "dim": 3, "metric": "l2",
         "maxdim": 1},
        # the headline workload: the front end of the symmetric kNN flag
        # complex of a 16-Gaussian mixture, host points in and host arrays out
        {"name": "knn_front_gmm100k", "op": "knn_front", "cloud": "gmm", "n": 100000, "dim": 32, "metric": "l2",
         "k": 15, "maxdim": 1},
        # the reference's published kNN workload: uniform points in R^3, k = 15
        {"name": "knn_graph_uniform100k", "op": "knn_graph", "cloud": "uniform", "n": 100000, "dim": 3,
         "metric": "l2", "k": 15},
        # ragged sizes and a metric without a contraction: lists only
        {"name": "knn_linf_20011x8", "op": "knn", "cloud": "gauss", "n": 20011, "dim": 8, "metric": "linf", "k": 10},
        # the mixture's kNN lists under a non-integer Minkowski metric
        {"name": "knn_lp_gmm100k", "op": "knn", "cloud": "gmm", "n": 100000, "dim": 32, "metric": "lp:1.5", "k": 15},
        # the reference's published threshold workload: uniform points in R^3,
        # tau = 0.105 (about 240 neighbours a point)
        {"name": "radius_uniform50k", "op": "radius", "cloud": "uniform", "n": 50000, "dim": 3, "metric": "l2",
         "tau": 0.105},
        # H0 of the complete graph on the mixture
        {"name": "mst_gmm100k", "op": "mst", "cloud": "gmm", "n": 100000, "dim": 32, "metric": "l2"},
        # the batched workload: 512 uneven noisy circles and figure-eights
        {"name": "batch_512", "op": "batch", "clouds": 512, "lo": 64, "hi": 2048, "metric": "l2"},
        # the differentiable workload: loss forward and backward, 64 clouds
        {"name": "topo_step_64x512", "op": "topo", "clouds": 64, "n": 512, "metric": "l2"},
        # the whole call on the reference's example: 1,000 points on a torus
        {"name": "persistence_torus1000", "op": "persistence", "cloud": "torus", "n": 1000, "dim": 3, "metric": "l2",
         "maxdim": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["dense", "dense", "knn", "knn", "knn_graph", "knn_front", "radius", "mst", "batch", "topo",
                     "persistence"])
    if op == "dense":
        cloud = rng.choice(["circle", "gauss", "uniform", "lattice", "torus"])
        dim = {"circle": 3, "torus": 3, "lattice": 4}.get(cloud) or rng.choice([2, 3, 4, 5, 8, 16, 24, 32])
        return {"op": op, "cloud": cloud, "n": _log(rng, 64, 12000), "dim": dim,
                "metric": rng.choice(["l2", "l2", "l1", "linf", "lp:1.5", "lp:3"]), "maxdim": rng.choice([1, 2])}
    if op in ("knn", "knn_graph"):
        metric = rng.choice(["l2", "l2", "l1", "linf", "lp:1.5", "lp:3"])
        dim = rng.choice([2, 3, 4, 5, 8, 10, 16, 24, 32, 50, 64])
        most = 100000 if dim <= 32 and not metric.startswith("lp") else 40000
        return {"op": op, "cloud": rng.choice(["gmm", "uniform", "gauss"]), "n": _log(rng, 1000, most), "dim": dim,
                "metric": metric, "k": rng.randint(1, 16)}
    if op == "knn_front":
        return {"op": op, "cloud": rng.choice(["gmm", "gauss"]), "n": _log(rng, 2000, 100000),
                "dim": rng.choice([3, 16, 32]), "metric": "l2", "k": rng.randint(4, 16), "maxdim": 1}
    if op == "radius":
        n, dim, metric = _log(rng, 1000, 50000), rng.choice([2, 3, 4]), rng.choice(["l2", "l2", "l1", "linf"])
        degree = rng.uniform(8, 200)   # of an interior point
        return {"op": op, "cloud": "uniform", "n": n, "dim": dim, "metric": metric,
                "tau": round((degree / (n * _ball(dim, metric))) ** (1 / dim), 5)}
    if op == "mst":
        dim = rng.choice([2, 3, 8, 16, 32])
        return {"op": op, "cloud": rng.choice(["gmm", "uniform"]), "n": _log(rng, 1000, 100000 if dim == 32 else 50000),
                "dim": dim, "metric": rng.choice(["l2", "l2", "l1", "linf"]) if dim < 32 else "l2"}
    if op == "batch":
        lo = rng.randint(32, 256)
        return {"op": op, "clouds": _log(rng, 8, 512), "lo": lo, "hi": _log(rng, lo + 64, 2048),
                "metric": rng.choice(["l2", "l2", "l1", "linf"])}
    if op == "topo":
        return {"op": op, "clouds": rng.randint(2, 64), "n": _log(rng, 48, 512),
                "metric": rng.choice(["l2", "l2", "l1", "linf"])}
    return {"op": "persistence", "cloud": "torus", "n": _log(rng, 100, 1000), "dim": 3,
            "metric": rng.choice(["l2", "l1", "linf"]), "maxdim": rng.choice([1, 2])}


# ---------------------------------------------------------------------------
# Inputs, and the caller's buffers that results of unknown length go to (zero
# past their end, as large as the result can get).
# ---------------------------------------------------------------------------
def _points(case, seed):
    n, dim, cloud = case["n"], case["dim"], case["cloud"]
    if cloud == "gmm":
        return synth.gmm(n, dim, seed=seed)
    if cloud == "lattice":
        return synth.lattice(n, seed=seed, dim=dim)
    if cloud == "torus":
        return synth.torus(n, seed=seed)
    if cloud == "circle":
        return synth.circles(1, n, seed=seed)[0]
    return synth.uniform(n, dim, seed) if cloud == "uniform" else synth.gauss(n, dim, seed)


def _sizes(case):
    """The batched workload's cloud sizes (synth.circle_batch's own for its 512 clouds)."""
    return np.random.default_rng(4).integers(case["lo"], case["hi"] + 1, case["clouds"])


def _batch_points(case, seed):
    """Noisy circles and figure-eights of those sizes, as synth.circle_batch makes them."""
    rng = np.random.default_rng(seed)
    out = []
    for m in _sizes(case):
        r = rng.uniform(0.5, 2)
        t = rng.uniform(0, 2 * np.pi, m)
        eight = rng.random() < 0.5
        side = np.where(rng.random(m) < 0.5, -r, r) if eight else 0.0
        y = np.c_[r * np.cos(t) + side, r * np.sin(t), np.zeros(m)]
        out.append((y + rng.normal(0, 0.03, y.shape)).astype(np.float32))
    return out


def _ball(dim, metric):
    """Volume of the metric's unit ball."""
    if metric == "linf":
        return 2.0 ** dim
    if metric == "l1":
        return 2.0 ** dim / math.factorial(dim)
    return math.pi ** (dim / 2) / math.gamma(dim / 2 + 1)


def _zeros(count, dtype, pinned=False):
    return torch.zeros(count, dtype=dtype).pin_memory() if pinned else torch.zeros(count, dtype=dtype, device="cuda")


def _graph_buffers(n, entries, pinned=False):
    return {"rp": _zeros(n + 1, torch.int64, pinned), "ci": _zeros(entries, torch.int32, pinned),
            "w": _zeros(entries, torch.float32, pinned)}


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "ctx": _ctx()}
    if op == "batch":
        clouds = _batch_points(case, seed)
        pairs = sum(len(c) * (len(c) - 1) // 2 for c in clouds)
        st["x"] = torch.from_numpy(np.concatenate(clouds)).cuda()
        st["batch"] = ops.DenseBatch(st["ctx"], [len(c) for c in clouds], 3, case["metric"])
        st["out"] = {"radius": _zeros(len(clouds), torch.float32), "edge_offset": _zeros(len(clouds) + 1, torch.int64),
                     "diam": _zeros(pairs, torch.float32), "verts": _zeros(2 * pairs, torch.int32)}
    elif op == "topo":
        clouds = synth.circles(case["clouds"], case["n"], seed=seed)
        st["sizes"] = np.array([len(c) for c in clouds], np.uint32)
        st["x"] = torch.from_numpy(np.concatenate(clouds)).cuda()
    elif op == "persistence":
        st["x"] = _points(case, seed)
    else:
        n = case["n"]
        x = torch.from_numpy(_points(case, seed))
        st["metric"] = capi.metric_parse(case["metric"])
        if op == "knn_front":
            st["x"] = x.pin_memory()
            m = 2 * n * case["k"]
            st["out"] = _graph_buffers(n, m, True) | {
                "h0": _zeros(n, torch.float32, True), "cidx": _zeros(m, torch.int64, True),
                "cd": _zeros(m, torch.float32, True), "cf": _zeros(m, torch.int64, True),
                "ca": _zeros(m, torch.uint8, True)}
        else:
            st["x"] = x.cuda()
        if op == "knn_graph":
            st["out"] = _graph_buffers(n, 2 * n * case["k"])
        elif op == "radius":
            degree = n * _ball(case["dim"], case["metric"]) * case["tau"] ** case["dim"]
            st["out"] = _graph_buffers(n, min(n * n, int(1.1 * n * degree) + 8192))
        elif op == "dense":
            m = n * (n - 1) // 2
            st["out"] = {"mat": torch.zeros((n, n), dtype=torch.float32, device="cuda"),
                         "keys": _zeros(m, torch.int64), "app": _zeros(m, torch.uint8), "tree": _zeros(m, torch.uint8),
                         "cidx": _zeros(m, torch.int64), "cd": _zeros(m, torch.float32), "cf": _zeros(m, torch.int64),
                         "ca": _zeros(m, torch.uint8), "h0": _zeros(n, torch.float32)}
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
def run(st):
    case, ctx = st["case"], st["ctx"]
    op = case["op"]
    if op == "dense":
        return _dense(st)
    if op == "knn":
        ids, d = ops.knn(ctx, st["x"], case["k"], case["metric"])
        return {"ids": ids, "d": d}
    if op in ("knn_graph", "radius"):
        return _graph(st)
    if op == "mst":
        return {"deaths": ops.mst_deaths(ctx, st["x"], case["metric"])}
    if op == "knn_front":
        return _knn_front(st)
    if op == "batch":
        return _batch(st)
    if op == "topo":
        x = st["x"].detach().requires_grad_(True)
        loss = topo.topo_loss(x, st["sizes"], case["metric"])
        loss.backward()
        return {"loss": loss.detach(), "grad": x.grad}
    dgms, info = tg.persistence(st["x"], maxdim=case["maxdim"], metric=case["metric"])
    bars = np.zeros((len(dgms), 4 * case["n"], 2), np.float32)
    for d, g in enumerate(dgms):
        bars[d, :len(g)] = g
    return {"bars": bars, "count": np.array([len(g) for g in dgms]), "threshold": info["threshold"]}


def _take(ctx, buf, addr, count):
    """`count` entries of the context's device array at `addr` into the caller's buffer."""
    if count > buf.numel():
        raise RuntimeError("the caller's buffer is too small")
    if count:
        ctx.check(ctx.L.tt_copy_async(ctx.h, buf.data_ptr(), addr, count * buf.element_size()))


def _dense(st):
    case, ctx, out = st["case"], st["ctx"], st["out"]
    kind, p = st["metric"]
    n = case["n"]
    radius, r = ctypes.c_float(), capi.Dim0Out()
    ctx.check(ctx.L.tt_dense_distances(ctx.h, st["x"].data_ptr(), n, case["dim"], kind, p, out["mat"].data_ptr(),
                                       ctypes.byref(radius)))
    ctx.check(ctx.L.tt_dim0(ctx.h, out["mat"].data_ptr(), None, None, None, n, radius.value, case["maxdim"],
                            ctypes.byref(r)))
    _take(ctx, out["keys"], r.edge_keys_dev, r.edges)
    _take(ctx, out["app"], r.apparent_dev, r.edges)
    _take(ctx, out["tree"], r.tree_dev, r.edges)
    _take(ctx, out["cidx"], r.col_index_dev, r.columns)
    _take(ctx, out["cd"], r.col_diameter_dev, r.columns)
    _take(ctx, out["cf"], r.col_cofacet_dev, r.columns)
    _take(ctx, out["ca"], r.col_cofacet_app_dev, r.columns)
    _take(ctx, out["h0"], r.h0_death_dev, r.h0_finite)
    return out | {"radius": radius.value, "edges": r.edges, "columns": r.columns, "essential": r.essential}


def _graph(st):
    case, ctx, out = st["case"], st["ctx"], st["out"]
    kind, p = st["metric"]
    g = capi.CsrOut()
    if case["op"] == "radius":
        ctx.check(ctx.L.tt_radius_graph(ctx.h, st["x"].data_ptr(), case["n"], case["dim"], kind, p, case["tau"],
                                        ctypes.byref(g)))
    else:
        ctx.check(ctx.L.tt_knn_graph(ctx.h, st["x"].data_ptr(), case["n"], case["dim"], kind, p, case["k"],
                                     ctypes.byref(g)))
    _take(ctx, out["rp"], g.row_ptr_dev, g.n + 1)
    _take(ctx, out["ci"], g.col_dev, g.nnz)
    _take(ctx, out["w"], g.weight_dev, g.nnz)
    return out | {"nnz": g.nnz}


def _knn_front(st):
    case, ctx, out = st["case"], st["ctx"], st["out"]
    kind, p = st["metric"]
    u64, ref = ctypes.c_uint64, ctypes.byref
    nnz, nh0, essential, columns, edges = u64(), u64(), u64(), u64(), u64()
    cap = out["ci"].numel()
    ctx.check(ctx.L.tt_knn_front_h(
        ctx.h, st["x"].data_ptr(), case["n"], case["dim"], kind, p, case["k"], case["maxdim"], out["rp"].data_ptr(),
        out["ci"].data_ptr(), out["w"].data_ptr(), cap, ref(nnz), out["h0"].data_ptr(), ref(nh0), ref(essential),
        out["cidx"].data_ptr(), out["cd"].data_ptr(), out["cf"].data_ptr(), out["ca"].data_ptr(), cap, ref(columns),
        ref(edges)))
    return out | {"nnz": nnz.value, "columns": columns.value, "essential": essential.value, "edges": edges.value}


def _batch(st):
    ctx, out, b = st["ctx"], st["out"], st["batch"]
    b.load(st["x"])
    b.run()
    r = capi.BatchOut()
    ctx.check(ctx.L.tt_batch_result(b.h, ctypes.byref(r)))
    _take(ctx, out["radius"], r.radius_dev, r.clouds)
    _take(ctx, out["edge_offset"], r.edge_offset_dev, r.clouds + 1)
    m = int(out["edge_offset"][-1])
    _take(ctx, out["diam"], r.diam_dev, m)
    _take(ctx, out["verts"], r.verts_dev, 2 * m)
    return out


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def work(case):
    op = case["op"]
    if op == "batch":
        mean = (case["lo"] + case["hi"]) / 2
        square = mean * mean + (case["hi"] - case["lo"]) ** 2 / 12   # E[n^2] of the uniform sizes
        pairs = case["clouds"] * square / 2
        # the points, the matrices (4 B an entry), the edges (4 B length, 8 B
        # ends); about four pairs in five lie within the enclosing radius
        return {"bytes": case["clouds"] * mean * 12 + 8 * pairs + 0.8 * 12 * pairs, "flops": 9 * pairs}
    if op == "topo":
        n, c = case["n"], case["clouds"]
        return {"bytes": c * n * 24, "flops": 9 * c * n * n / 2}
    n, dim = case["n"], case["dim"]
    pts = 4 * n * dim
    if op == "dense":
        pairs = n * (n - 1) / 2
        # the matrix, then key and two flags for the kept edges (about half)
        return {"bytes": pts + 4 * n * n + 0.5 * 10 * pairs, "flops": 3 * dim * pairs}
    if op == "persistence":
        return {"bytes": pts + 8 * n, "flops": 3 * dim * n * (n - 1) / 2}
    if op == "mst":
        return {"bytes": pts + 4 * n, "flops": 3 * dim * n}
    if op == "radius":
        m = n * n * _ball(dim, case["metric"]) * case["tau"] ** dim
        return {"bytes": pts + 8 * n + 8 * m, "flops": 3 * dim * m}
    k = case["k"]
    if op == "knn":
        return {"bytes": pts + 8 * n * k, "flops": 3 * dim * n * k}
    # a graph holds about 1.6 entries a list entry once mutual ones coincide
    graph = 8 * n + 8 * 1.6 * n * k
    if op == "knn_graph":
        return {"bytes": pts + graph, "flops": 3 * dim * n * k}
    return {"bytes": pts + graph + 4 * n + 21 * 0.7 * n * k, "flops": 3 * dim * n * k}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits.
# ---------------------------------------------------------------------------
def _p(metric):
    return {"l1": 1.0, "l2": 2.0, "linf": math.inf}.get(metric) or float(metric[3:])


def _cdist(a, b, p):
    return torch.cdist(a, b, p=p, compute_mode="donot_use_mm_for_euclid_dist")


def _tree_weights(x, p):
    """Sorted minimum-spanning-tree weights, one vertex at a time."""
    n = x.shape[0]
    near = torch.full((n,), math.inf, dtype=torch.float64, device=x.device)
    done = torch.zeros(n, dtype=torch.float64, device=x.device)   # +inf once in the tree
    cur = torch.zeros(1, dtype=torch.int64, device=x.device)
    got = torch.empty(n, dtype=torch.float64, device=x.device)
    for step in range(n - 1):
        done.index_fill_(0, cur, math.inf)
        near = torch.minimum(near, torch.linalg.vector_norm(x - x.index_select(0, cur), ord=p, dim=1))
        best, at = torch.min(near + done, 0)
        got[step] = best
        cur = at.view(1)
    return got[: n - 1].sort().values


def exact(case, seed):
    op, metric = case["op"], case.get("metric")
    if op in ("radius", "knn_graph", "knn_front", "topo", "persistence"):
        return None   # which pairs an output holds hangs on ties and thresholds of the 32-bit distances
    p = _p(metric)
    if op == "batch":
        radius = []
        for c in _batch_points(case, seed):
            x = torch.from_numpy(c).cuda().double()
            radius.append(_cdist(x, x, p).max(1).values.min())
        return {"radius": torch.stack(radius), "edge_offset": None, "diam": None, "verts": None}
    x = torch.from_numpy(_points(case, seed)).cuda().double()
    n = x.shape[0]
    if op == "dense":
        mat = _cdist(x, x, p)
        out = {k: None for k in ("keys", "app", "tree", "cidx", "cd", "cf", "ca", "edges", "columns", "essential")}
        out["h0"] = torch.cat([_tree_weights(x, p), x.new_zeros(1)])
        out["mat"], out["radius"] = mat, float(mat.max(1).values.min())
        return out
    if op == "mst":
        return {"deaths": _tree_weights(x, p)}
    if metric.startswith("lp") and n * n * case["dim"] > 1e11:
        return None
    d = torch.empty((n, case["k"]), dtype=torch.float64, device=x.device)
    rows = max(1, (1 << 27) // n)
    for i in range(0, n, rows):
        part = _cdist(x[i:i + rows], x, p)
        r = torch.arange(part.shape[0], device=x.device)
        part[r, r + i] = math.inf
        d[i:i + rows] = torch.topk(part, case["k"], dim=1, largest=False, sorted=True).values
    return {"ids": None, "d": d}
