"""Timed cases over the public entry points: exact and reference-parity range batches, exact KNN, the
per-level plugin and the index build, from one query at a time to the batched configuration.

A case is a dict of plain values. `prepare` makes what a program holds before the call (the prepared
handle, which it keeps over all its batches, and new queries or points drawn from the seed), `run`
makes one call and returns its outputs, `work` counts what the call cannot do without, and `exact`
gives the computed numbers in 64 bits from the index's own arrays by brute force.

Indexes are the seeded synthetic ones of the benchmark configurations (`workloads.CONFIGS`), some at
a smaller N; queries follow the same distributions (boxes and points around data points).
"""
import collections
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "tblaeq_b200" not in sys.modules:
        d = os.path.join(_ROOT, "t-blaeq_b200")
        spec = importlib.util.spec_from_file_location("tblaeq_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tblaeq_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tblaeq_b200"]


def _index(N, D, ratios="100,50,20", gseed=1, sigma=3.0):
    return dict(N=N, D=D, ratios=ratios, gseed=gseed, sigma=sigma)


_SMALL = _index(500_000, 5, "80,40,20", 20260330, 2.2)
_BATCHED = _index(10_000_000, 8)
_HIGH = _index(5_000_000, 16, "100,50,20", 2, 2.5)


def listed():
    return [
        # One box at a time on the small configuration: the reference's own calling pattern
        # (performSingleRangeQuery), all latency.
        dict(name="range_one", kind="range", nq=1, hw_lo=0.05, hw_hi=0.05, entry="host", **_SMALL),
        # The small configuration's 100 boxes as one batch.
        dict(name="range_small", kind="range", nq=100, hw_lo=0.05, hw_hi=0.05, entry="host", **_SMALL),
        # The batched range configuration end to end: host boxes in, offsets and ids out.
        dict(name="range_batch", kind="range", nq=4096, hw_lo=0.001, hw_hi=0.1, entry="host", **_BATCHED),
        # The same index, a few ragged boxes as a serving lane collects them between two batches.
        dict(name="range_lane", kind="range", nq=37, hw_lo=0.001, hw_hi=0.05, entry="host", **_BATCHED),
        # Large answers with their coordinates, left on the device for the caller's next kernel; an
        # odd dimension.
        dict(name="range_vals", kind="range", nq=301, hw_lo=0.02, hw_hi=0.1, entry="vals", **_index(1_500_000, 3)),
        # The reference's candidate sets, as a program that replaces the reference asks for them.
        dict(name="range_ref", kind="range", nq=100, hw_lo=0.05, hw_hi=0.05, entry="ref", **_SMALL),
        # One KNN query through the per-level plugin (IQueryStrategy::runLevel), level by level.
        dict(name="plugin_knn", kind="plugin", nq=1, k_lo=10, k_hi=10, noise=0.01, **_SMALL),
        # One exact KNN query at a time.
        dict(name="knn_one", kind="knn", nq=1, k_lo=10, k_hi=10, noise=0.01, learned=False, **_BATCHED),
        # A serving lane's KNN batch: per-query K log-uniform in [1, 256].
        dict(name="knn_lane", kind="knn", nq=300, k_lo=1, k_hi=256, noise=0.01, learned=False, **_BATCHED),
        # The batched KNN leg: 4,096 points, K = 20 and 100 in turn.
        dict(name="knn_batch", kind="knn", nq=4096, k_lo=20, k_hi=100, noise=0.02, learned=False, **_BATCHED),
        # High-dimensional KNN with the trained frontier scorer.
        dict(name="knn_d16", kind="knn", nq=1000, k_lo=20, k_hi=100, noise=0.02, learned=True, **_HIGH),
        # Building an index from points: k-means per level, then the assembly.
        dict(name="build", kind="build", N=1_000_000, D=16, ratios="100,50,20", iters=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["range", "range", "range", "knn", "knn", "build", "plugin"])
    if kind == "build":
        D = rng.choice([3, 5, 8, 11, 16])
        return dict(kind="build", N=_log(rng, 20_000, 1_000_000), D=D, ratios=rng.choice(["100,50,20", "80,40,20"]),
                    iters=rng.choice([5, 10, 20]))
    if kind == "range":
        D = rng.choice([2, 3, 4, 5, 6, 7, 8, 8, 12, 16])
        entry = rng.choice(["host", "host", "host", "vals", "ref"])
        # Low dimensions and the reference's candidate sets answer with a large share of the index:
        # fewer and smaller boxes there, as no call may outgrow the largest listed one.
        big = entry == "ref" or D < 6
        N = _log(rng, 100_000, 500_000 if big else 10_000_000 if D <= 8 else 4_000_000)
        nq = _log(rng, 1, 100 if entry == "ref" or D == 2 else 300 if big else 4096)
        return dict(kind="range", nq=nq, hw_lo=rng.choice([0.001, 0.01]), hw_hi=rng.choice([0.03, 0.05, 0.1]),
                    entry=entry, **_index(N, D, rng.choice(["100,50,20", "80,40,20"]), rng.randrange(1, 1000)))
    D = rng.choice([2, 3, 5, 8, 8, 10, 16])
    N = _log(rng, 100_000, 500_000 if kind == "plugin" else 10_000_000 if D <= 8 else 2_000_000)
    most = 1 if kind == "plugin" else 4096 if D <= 8 else 1000
    k_lo = _log(rng, 1, 20)
    c = dict(kind=kind, nq=_log(rng, 1, most), k_lo=k_lo, k_hi=max(k_lo, _log(rng, 1, 256)),
             noise=rng.choice([0.01, 0.02]), **_index(N, D, rng.choice(["100,50,20", "80,40,20"]), rng.randrange(1, 1000)))
    return c if kind == "plugin" else dict(c, learned=False)


def _ratios(case):
    return tuple(int(r) for r in case["ratios"].split(","))


# Prepared handles, the last two used: a program opens an index once and sends it many batches.
_handles = collections.OrderedDict()


def _handle(case):
    tb = _package()
    key = (case["N"], case["D"], case["ratios"], case["gseed"], case["sigma"], bool(case.get("learned")))
    if key not in _handles:
        while len(_handles) >= 2:
            _handles.popitem(last=False)
        r = _ratios(case)
        h = tb.QueryHandler.generate(case["N"], case["D"], 1.0, 100.0, False, len(r) + 1, r, case["gseed"], case["sigma"])
        h.prepare_for_query(tb.LevelPolicy.L0)
        lo, hi = _extent(h)
        if case.get("learned"):
            rng = np.random.default_rng(99)
            h.scorer_train(_points(h, case, rng, 512, hi - lo), K=40, max_samples=20000, epochs=2, seed=1)
        _handles[key] = (h, hi - lo)
    _handles.move_to_end(key)
    return _handles[key]


def _extent(h):
    """Extent of a fixed sample of the data points, which boxes and noise scale with."""
    pts, _ = h.decode_points(np.random.default_rng(7).integers(0, h.info()["N"], 65536))
    return pts.min(axis=0), pts.max(axis=0)


def _points(h, case, rng, n, ext):
    centres, _ = h.decode_points(rng.integers(0, case["N"], n))
    return np.ascontiguousarray(centres + rng.normal(0.0, 1.0, centres.shape) * (case["noise"] * ext))


def _boxes(h, case, rng, ext):
    n, D = case["nq"], case["D"]
    centres, _ = h.decode_points(rng.integers(0, case["N"], n))
    hw = np.exp(rng.uniform(math.log(case["hw_lo"]), math.log(case["hw_hi"]), (n, D))) * ext
    return np.ascontiguousarray(np.concatenate([centres - hw, centres + hw], axis=1))


def _wanted(case):
    """Neighbours per query, of the case and not of the seed (the answer's size follows from them):
    k_lo and k_hi in turn when both are of one order, else log-uniform."""
    n, a, b = case["nq"], case["k_lo"], case["k_hi"]
    rng = np.random.default_rng(n)
    if a == b:
        return a
    if b <= 5 * a:
        return np.where(np.arange(n) % 2 == 0, a, b).astype(np.uint32)
    return np.floor(np.exp(rng.uniform(math.log(a), math.log(b), n))).astype(np.uint32)


def _dataset(case, seed):
    """Clustered FP32 points: 80% in Gaussian clusters, 20% uniform, coordinates in [1, 100]."""
    rng = np.random.default_rng(seed)
    N, D = case["N"], case["D"]
    m = max(1, N // 5000)
    X = rng.uniform(1.0, 100.0, (N, D)).astype(np.float32)
    n = int(0.8 * N)
    c = rng.uniform(2.0, 99.0, (m, D)).astype(np.float32)
    X[:n] = c[rng.integers(0, m, n)] + rng.standard_normal((n, D), dtype=np.float32)
    np.clip(X, 1.0, 100.0, out=X)
    return X[rng.permutation(N)]


def _room(case):
    """Rows of the caller's answer buffers: range answers and candidate sets vary with the query."""
    if case["kind"] == "plugin":
        return case["N"]
    return 1 << (18 if case["entry"] == "host" else 22)


def prepare(case, seed):
    s = dict(case=case)
    if case["kind"] == "build":
        s["X"] = _dataset(case, seed)
        return s
    h, ext = _handle(case)
    rng = np.random.default_rng(seed)
    s["h"] = h
    if case["kind"] == "range":
        s["q"] = _boxes(h, case, rng, ext)
        if case["entry"] != "host":
            s["dq"] = torch.from_numpy(s["q"]).cuda()
            s["ids"] = torch.zeros(_room(case), dtype=torch.int64, device="cuda")
            if case["entry"] == "vals":
                s["vals"] = torch.zeros((_room(case), case["D"]), dtype=torch.float64, device="cuda")
        else:
            s["ids"] = np.zeros(_room(case), np.uint64)
    else:
        s["q"] = _points(h, case, rng, case["nq"], ext)
        s["K"] = _wanted(case)
        if case["kind"] == "plugin":
            s["ids"] = torch.zeros(_room(case), dtype=torch.int64, device="cuda")
            s["vals"] = torch.zeros((_room(case), case["D"]), dtype=torch.float64, device="cuda")
    return s


def _fill(buf, rows):
    """Copies an answer into the caller's buffer (as much as it holds) and returns the buffer."""
    n = min(len(buf), len(rows))
    buf[:n] = rows[:n]
    return buf


def run(state):
    tb = _package()
    case = state["case"]
    if case["kind"] == "build":
        h, _ = tb.QueryHandler.build(state["X"], height=len(_ratios(case)) + 1, ratios=_ratios(case),
                                     iters=case["iters"], seed=1)
        n = len(_ratios(case))
        out = {"vals": [h.host_array(0, l) for l in range(n)], "cols": [h.host_array(1, l) for l in range(n)],
               "radius": [h.host_array(2, l) for l in range(n)], "map": [h.host_array(3, m) for m in range(1, n + 1)]}
        h.close()
        return out
    h = state["h"]
    if case["kind"] == "range":
        if case["entry"] == "host":
            offs, ids, _ = h.query_batch_host(tb.QueryType.RANGE, state["q"], tb.Mode.EXACT)
            return {"offsets": offs, "ids": _fill(state["ids"], ids)}
        vals = case["entry"] == "vals"
        r = h.query_batch(tb.QueryType.RANGE, state["dq"], tb.Mode.EXACT if vals else tb.Mode.REF_PARITY,
                          flags=tb.WANT_VALS if vals else 0)
        out = {"offsets": r.offsets.torch(), "ids": _fill(state["ids"], r.ids.torch().view(torch.int64))}
        return dict(out, vals=_fill(state["vals"], r.vals.torch())) if vals else out
    if case["kind"] == "plugin":
        g = h.coarsest_grid()
        for l in range(len(_ratios(case))):
            g = h.run_level(l, g, tb.QueryType.POINT, point=state["q"][0], K=case["k_lo"])
        ids = tb.DeviceArray(g.ids, (g.nnz,), "<u8").torch().view(torch.int64)
        vals = tb.DeviceArray(g.vals, (g.nnz, g.dim), "<f8").torch()
        return {"count": int(g.nnz), "ids": _fill(state["ids"], ids), "vals": _fill(state["vals"], vals)}
    offs, ids, d2 = h.query_batch_host(tb.QueryType.POINT, state["q"], tb.Mode.EXACT, K=state["K"])
    return {"offsets": offs, "ids": ids, "dist2": d2}


def work(case):
    """Bytes: the queries, and per answer the point's row and the written id (distance, coordinates);
    a box around a data point has one answer at least. Build: the points in, the index out, and the
    distance contraction of each level and iteration."""
    N, D = case["N"], case["D"]
    if case["kind"] == "build":
        flops, out, n = 0, 0, N
        for r in _ratios(case):
            k = max(1, n // r)
            flops += 2 * n * k * D * case["iters"]
            out += n * (8 * D + 8) + k * 16
            n = k
        return {"bytes": 4 * N * D + out, "flops": flops}
    nq = case["nq"]
    if case["kind"] == "range":
        return {"bytes": nq * (16 * D + 8) + nq * (8 * D + 8 + (8 * D if case["entry"] == "vals" else 0)), "flops": 0}
    k = nq * 0.5 * (case["k_lo"] + case["k_hi"])
    return {"bytes": nq * (8 * D + 8) + k * (8 * D + 16), "flops": 3 * k * D}


def _decoded(h, case):
    """(points, in the order a traversal meets them) from the index's arrays: a node's coordinates
    are its row of the P tensor times its parent's, its children the rows of its column."""
    D, L = case["D"], len(_ratios(case))
    x = h.host_array(5).reshape(-1, D)
    node = h.host_array(4).astype(np.int64)
    for l in range(L):
        P = h.host_array(0, l).reshape(-1, D)
        col = h.host_array(1, l).astype(np.int64)
        n = col[node + 1] - col[node]
        first = np.cumsum(n) - n
        rows = np.arange(int(n.sum())) + np.repeat(col[node] - first, n)
        x = P[rows] * np.repeat(x, n, axis=0)
        node = h.host_array(3, l + 1).astype(np.int64)[rows]
    return x


def exact(case, seed):
    if case["kind"] not in ("knn", "range") or (case["kind"] == "range" and case["entry"] != "vals"):
        return None  # whole numbers, and the reference's candidate sets and builds, which have no other value
    s = prepare(case, seed)
    x = torch.from_numpy(_decoded(s["h"], case)).cuda()
    q = torch.from_numpy(s["q"]).cuda()
    D = case["D"]
    if case["kind"] == "range":
        if D in (4, 8, 16):
            return None  # there the points of a cluster come in an order of the index's own
        vals = [x[((x >= b[:D]) & (x <= b[D:])).all(1)] for b in q]
        return {"offsets": None, "ids": None, "vals": _fill(torch.zeros_like(s["vals"]), torch.cat(vals))}
    if case["nq"] * case["N"] > 5e10:
        return None
    K = np.broadcast_to(np.asarray(s["K"]), (case["nq"],))
    xt = x.t().contiguous()
    step = max(1, int(4e8 // case["N"]))
    d2 = []
    for i in range(0, case["nq"], step):
        d = torch.zeros((min(step, case["nq"] - i), case["N"]), dtype=torch.float64, device="cuda")
        for j in range(D):
            t = q[i:i + step, j:j + 1] - xt[j]
            d.addcmul_(t, t)
        top = torch.topk(d, int(min(K.max(), case["N"])), dim=1, largest=False).values
        d2 += [top[r, :int(K[i + r])] for r in range(top.shape[0])]
    return {"offsets": None, "ids": None, "dist2": torch.cat(d2)}
