"""Performance cases of the framework: the calls its users make, by their public entry points.

A case is a dict of plain values. ``kind`` names the entry point:

* ``call``: ``rips_persistence`` on one point cloud resident on the GPU;
* ``batch``: ``rips_persistence_batch`` on many clouds of uneven size and dimension;
* ``serve``: a burst of requests through a ``PersistenceServer`` that the program keeps;
* ``threshold``: ``auto_threshold`` and ``enclosing_radius`` on one cloud.

Clouds are i.i.d. N(0, 1) (``shape`` "normal") or noisy Clifford tori (``shape``
"torus"). The threshold of a call is ``t`` where it is positive, else the 95th
percentile of the 20-NN distances (``t`` 0: what ``auto_threshold`` estimates by
default), else the length that gives ``degree`` neighbours a point on average
(``t`` < 0). Requests over the reference's simplex limits are answered with its
ValueError, as a user's program meets it; the outputs then hold the simplex count
that it tells. The program collects H1 and H2 rows, whose number the data decide, in
buffers of its own (unused rows are NaN).
"""
from __future__ import annotations

import math
import os
import re
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "flash-ph_b200"))

from flashph_b200 import auto_threshold, enclosing_radius, rips_persistence  # noqa: E402
from flashph_b200.batch import rips_persistence_batch  # noqa: E402
from flashph_b200.serve import PersistenceServer  # noqa: E402

DEVICE = "cuda"
MAX_TRIANGLES = 10_000_000  # the reference's default limit of a call


def _call(n, d, max_dim, t, shape="normal", degree=0.0):
    return {"kind": "call", "n": n, "d": d, "max_dim": max_dim, "t": t, "shape": shape, "degree": degree}


def listed():
    """The listed cases, the smallest calls first."""
    cases = [
        # an exploratory call on a small sampled surface with the default threshold: latency is all
        ("torus_211", _call(211, 4, 1, 0.0, "torus")),
        # the small plain configuration (H0-H2 of 500 points)
        ("small_h2", _call(500, 10, 2, 2.8)),
        # a scan's 3-D points, odd size, default threshold, below the tensor-core screen's dimensions
        ("scan_3d", _call(4001, 3, 1, 0.0, "torus")),
        # the headline: a large sparse complex up to H2
        ("sparse_20k", _call(20000, 10, 2, 1.4)),
        # the same at ten times the points, H1
        ("sparse_200k", _call(200000, 10, 1, 1.1)),
        # high-dimensional embeddings: all pairs screened on the tensor cores
        ("precision_200k", _call(200000, 50, 1, 6.0)),
        # single-linkage (H0 alone) of a large planar set
        ("h0_plane", _call(50021, 2, 0, -1.0, degree=12.0)),
        # a dense complex of a mid-size cloud at the default threshold (millions of triangles)
        ("dense_h1", _call(1501, 8, 1, 0.0)),
        # a dense H2 request (millions of tetrahedra)
        ("dense_h2", _call(331, 50, 2, 0.0)),
        # choosing the threshold of a cloud before the call
        ("thresholds_20k", {"kind": "threshold", "n": 20011, "d": 10, "k": 20, "shape": "normal"}),
        # a data set of many clouds of uneven size, all diagrams in one call
        ("batch_192", {"kind": "batch", "count": 192, "max_n": 4096}),
        # a burst of mixed requests at a server that runs for good
        ("serve_24", {"kind": "serve", "count": 24, "max_n": 50000}),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["sparse", "sparse", "sparse", "auto", "auto", "dense_h2", "threshold", "batch", "serve"])
    if kind == "sparse":
        d = rng.choice([2, 3, 4, 7, 8, 10, 17, 32, 50])
        n = int(_log(rng, 100, 200_000))
        degree = _log(rng, 1.0, 8.0 if d < 8 else 3.0)
        max_dim = rng.choice([0, 1, 1, 2]) if n < 65536 else rng.choice([0, 1, 1])
        return _call(n, d, max_dim, -1.0, degree=degree)
    if kind == "auto":
        shape = rng.choice(["normal", "torus"])
        return _call(int(_log(rng, 64, 4096 if shape == "torus" else 1500)), rng.choice([3, 4, 8, 32]), 1, 0.0, shape)
    if kind == "dense_h2":
        return _call(int(_log(rng, 64, 340)), rng.choice([4, 10, 50]), 2, 0.0)
    if kind == "threshold":
        return {"kind": "threshold", "n": int(_log(rng, 500, 20_000)), "d": rng.choice([3, 10, 50]),
                "k": rng.choice([5, 20, 64]), "shape": "normal"}
    if kind == "batch":
        return {"kind": "batch", "count": int(_log(rng, 8, 160)), "max_n": int(_log(rng, 256, 4096))}
    return {"kind": "serve", "count": int(_log(rng, 4, 20)), "max_n": int(_log(rng, 1000, 40_000))}


# ---- inputs ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _cloud(n, d, shape, gen):
    """(n, d) float32: N(0, 1), or a Clifford torus with 0.02 noise, padded and rotated
    (below four dimensions the first d rotated coordinates)."""
    if shape == "normal":
        return torch.randn(n, d, device=DEVICE, generator=gen)
    w = max(d, 4)
    ang = torch.rand(2, n, device=DEVICE, generator=gen, dtype=torch.float64) * (2 * math.pi)
    p = torch.stack([ang[0].cos(), ang[0].sin(), ang[1].cos(), ang[1].sin()], 1) / math.sqrt(2)
    p = p + 0.02 * torch.randn(n, 4, device=DEVICE, generator=gen, dtype=torch.float64)
    full = torch.zeros(n, w, device=DEVICE, dtype=torch.float64)
    full[:, :4] = p
    q = torch.linalg.qr(torch.randn(w, w, device=DEVICE, generator=gen, dtype=torch.float64))[0]
    return (full @ q.T)[:, :d].float().contiguous()


def _distances(a, b):
    return torch.cdist(a.double(), b.double(), compute_mode="donot_use_mm_for_euclid_dist")


def _knn(points, k, rows):
    """Distance of the given rows to their k-th nearest other point (64 bits)."""
    out = []
    step = max(1, (1 << 26) // points.shape[0])
    for part in rows.split(step):
        out.append(_distances(points[part], points).kthvalue(k + 1, dim=1).values)
    return torch.cat(out)


def _threshold(points, t, degree, gen):
    n = points.shape[0]
    if t > 0:
        return float(t)
    if t == 0:  # 95th percentile of the 20-NN distances, of a sample of the rows where there are many
        rows = torch.arange(n, device=DEVICE)
        if n > 4096:
            rows = torch.randperm(n, device=DEVICE, generator=gen)[:2048]
        return float(torch.quantile(_knn(points, min(20, n - 1), rows), 0.95))
    pairs = torch.randint(n, (2, 1 << 21), device=DEVICE, generator=gen)
    pairs = pairs[:, pairs[0] != pairs[1]]
    q = min(1.0, degree / (n - 1))
    m = pairs.shape[1]
    lengths = torch.cat([(points[a].double() - points[b].double()).norm(dim=1) for a, b in
                         zip(pairs[0].split(1 << 18), pairs[1].split(1 << 18))])
    return float(lengths.kthvalue(max(1, min(m, round(q * m)))).values)


def _sizes(case):
    """Log-uniform sizes of a batch or of a burst, in an order of no meaning."""
    lo, count = (100 if case["kind"] == "serve" else 64), case["count"]
    at = np.random.default_rng(count).permutation(count)
    return [int(lo * (case["max_n"] / lo) ** ((k + 0.5) / count)) for k in at]


def _requests(case, seed):
    """The clouds, thresholds and dimensions of a batch or of a burst."""
    gen = _generator(seed)
    clouds, ts, dims = [], [], []
    serve = case["kind"] == "serve"
    for c, n in enumerate(_sizes(case)):
        d = ([4, 10, 50] if serve else [3, 8, 32])[c % 3]
        clouds.append(_cloud(n, d, "normal" if serve or c % 2 == 0 else "torus", gen))
        ts.append(_threshold(clouds[-1], 0.0, 0.0, gen))
        dims.append(2 if serve and c % 5 == 1 else 1)
    return clouds, ts, dims


_server = None


def _the_server():
    """The server that a program keeps for its requests."""
    global _server
    if _server is None:
        _server = PersistenceServer()
    return _server


def _buffers(n, max_dim):
    """Where the program collects the rows of each dimension: n of H0, room for 8 a point of H1, 16 of H2."""
    return [torch.full((n * (8 * k or 1), 2), math.nan, device=DEVICE) for k in range(max_dim + 1)]


def prepare(case, seed):
    if case["kind"] in ("batch", "serve"):
        clouds, ts, dims = _requests(case, seed)
        return {"kind": case["kind"], "clouds": clouds, "t": ts, "max_dim": dims,
                "rows": _buffers(sum(_sizes(case)), max(dims)),
                "server": _the_server() if case["kind"] == "serve" else None}
    gen = _generator(seed)
    points = _cloud(case["n"], case["d"], case["shape"], gen)
    if case["kind"] == "threshold":
        return {"kind": "threshold", "points": points, "k": case["k"]}
    return {"kind": "call", "points": points, "max_dim": case["max_dim"],
            "rows": _buffers(case["n"], case["max_dim"]),
            "t": _threshold(points, case["t"], case["degree"], gen)}


# ---- one pass -------------------------------------------------------------------------
def _simplices(error):
    """The simplex count that the limit's ValueError tells."""
    return int(re.search(r"count (\d+)", str(error)).group(1))


def _collect(diagrams, buffer):
    """The rows of one or more diagrams at the head of the program's buffer."""
    total = sum(d.shape[0] for d in diagrams)
    if total > buffer.shape[0]:
        return torch.cat(diagrams)
    if len(diagrams) == 1:
        buffer[:total].copy_(diagrams[0])
    elif diagrams:
        torch.cat(diagrams, out=buffer[:total])
    return buffer


def _gather(results, dims, buffers):
    """The diagrams of many requests by dimension, each request's row counts, and the simplex counts of
    those over a limit."""
    done = [not isinstance(r, Exception) for r in results]
    out = {"count": np.array([[r[k].shape[0] if ok and k < len(r) else 0 for k in range(3)]
                              for r, ok in zip(results, done)], dtype=np.int64),
           "over": np.array([0 if ok else _simplices(r) for r, ok in zip(results, done)], dtype=np.int64)}
    for k, buffer in enumerate(buffers):
        out["h%d" % k] = _collect([r[k] for r, m, ok in zip(results, dims, done) if ok and m >= k], buffer)
    return out


def _answer(future):
    try:
        return future.result()
    except ValueError as ex:  # over one of the reference's limits
        return ex


def run(state):
    kind = state["kind"]
    if kind == "threshold":
        return {"auto": auto_threshold(state["points"], k=state["k"]), "radius": enclosing_radius(state["points"])}
    if kind == "batch":
        results = rips_persistence_batch(state["clouds"], state["t"], state["max_dim"])
        return _gather(results, state["max_dim"], state["rows"])
    if kind == "serve":
        futures = [state["server"].submit(*req) for req in zip(state["clouds"], state["t"], state["max_dim"])]
        return _gather([_answer(f) for f in futures], state["max_dim"], state["rows"])
    try:
        diagrams = rips_persistence(state["points"], state["t"], max_dim=state["max_dim"])
    except ValueError as ex:
        return {"over": _simplices(ex)}
    out = {"h0": diagrams[0]}
    for k, rows in enumerate(diagrams[1:], 1):
        out["h%d" % k] = _collect([rows], state["rows"][k])
        out["count%d" % k] = rows.shape[0]
    return out


def work(case):
    """Every pair's distance (a subtraction, a multiplication and an addition a coordinate), the points
    read once and the H0 rows written once (how many H1 and H2 rows there are is known only afterwards)."""
    if case["kind"] in ("batch", "serve"):
        n = _sizes(case)
        d = [([4, 10, 50] if case["kind"] == "serve" else [3, 8, 32])[c % 3] for c in range(len(n))]
        return {"bytes": sum(m * (4.0 * k + 8) for m, k in zip(n, d)),
                "flops": sum(1.5 * k * m * (m - 1) for m, k in zip(n, d))}
    n, d = case["n"], case["d"]
    passes = 2 if case["kind"] == "threshold" else 1
    return {"bytes": n * (4.0 * d + 8) * passes, "flops": 1.5 * d * n * (n - 1) * passes}


# ---- the same in 64 bits --------------------------------------------------------------
def _h0(points, t):
    """(0, death) rows ascending, then the essential ones: Boruvka on the full distance matrix."""
    n = points.shape[0]
    dist = _distances(points, points)
    dist.fill_diagonal_(math.inf)
    dist[dist >= t] = math.inf
    label = torch.arange(n, device=DEVICE)
    deaths = []
    while True:
        best, to = dist.min(dim=1)
        least = torch.full((n,), math.inf, device=DEVICE, dtype=torch.float64)
        least.scatter_reduce_(0, label, best, "amin")
        own = torch.nonzero(torch.isfinite(best) & (best == least[label])).flatten()
        if not own.numel():
            break
        # one edge a component; two components that chose the same edge count it once
        hook = torch.arange(n, device=DEVICE)
        hook[label[own]] = label[to[own]]
        root = torch.arange(n, device=DEVICE)
        mutual = (hook[hook] == root) & (hook != root)
        deaths.append(least[(hook != root) & ~(mutual & (root > hook))])
        hook = torch.where(mutual & (root < hook), root, hook)
        while not torch.equal(hook, hook[hook]):
            hook = hook[hook]
        label = hook[label]
        step = max(1, (1 << 27) // n)
        for a in range(0, n, step):
            part = dist[a:a + step]
            part[label[a:a + step, None] == label[None]] = math.inf
    deaths = torch.cat(deaths + [torch.full((0,), 0.0, device=DEVICE, dtype=torch.float64)]).sort().values
    rows = torch.zeros(n, 2, device=DEVICE, dtype=torch.float64)
    rows[:deaths.numel(), 1] = deaths
    rows[deaths.numel():, 1] = math.inf
    return rows


def _h1(points, t, most_edges=20_000, most_triangles=100_000):
    """(birth, death) rows by birth, by reduction of the triangles' boundaries; None for large complexes."""
    n = points.shape[0]
    if n > 2000:
        return None
    dist = _distances(points, points)
    i, j = torch.nonzero((dist < t).triu(1), as_tuple=True)
    order = dist[i, j].argsort(stable=True)
    i, j = i[order], j[order]
    m = i.numel()
    if not 0 < m <= most_edges:
        return None
    rank = torch.full((n, n), m, device=DEVICE, dtype=torch.int64)
    rank[i, j] = torch.arange(m, device=DEVICE)
    rank = torch.minimum(rank, rank.T)
    tri = []
    for e in torch.arange(m, device=DEVICE).split(1024):
        a, b = rank[i[e]], rank[j[e]]
        # the triangles whose last edge this is
        at, w = torch.nonzero((a < e[:, None]) & (b < e[:, None]), as_tuple=True)
        tri.append(torch.stack([e[at], a[at, w], b[at, w]], 1))
    tri = torch.cat(tri)
    if tri.shape[0] > most_triangles:
        return None
    length = dist[i, j].tolist()
    # positive edges close a cycle; a triangle's reduced boundary ends at the cycle's youngest edge
    parent = list(range(n))

    def find(v):
        while parent[v] != v:
            parent[v] = parent[parent[v]]
            v = parent[v]
        return v

    positive = []
    for e, (u, v) in enumerate(zip(i.tolist(), j.tolist())):
        u, v = find(u), find(v)
        if u == v:
            positive.append(e)
        parent[u] = v
    reduced, death = {}, {}
    for column in tri.tolist():
        last, column = column[0], set(column)
        while column:
            low = max(column)
            if low not in reduced:
                reduced[low], death[low] = column, last
                break
            column = column ^ reduced[low]
    rows = [(length[e], length[death[e]] if e in death else math.inf) for e in positive if death.get(e) != e]
    return torch.tensor(rows, dtype=torch.float64, device=DEVICE).reshape(-1, 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None  # its largest clouds take too long this way
    if kind == "batch":
        clouds, ts, _ = _requests(case, seed)
        rows = []
        for points, t in zip(clouds, ts):
            near = (_distances(points, points) < t).fill_diagonal_(False).float()
            if float(((near @ near) * near).double().sum()) / 6 <= MAX_TRIANGLES:
                rows.append(_h0(points, t))
        buffer = _buffers(sum(_sizes(case)), 0)[0].double()
        return {"count": None, "over": None, "h0": _collect(rows, buffer), "h1": None}
    state = prepare(case, seed)
    points = state["points"]
    n = points.shape[0]
    if kind == "threshold":
        knn = _knn(points, state["k"], torch.arange(n, device=DEVICE))
        far = torch.cat([_distances(p, points).amax(dim=1) for p in points.split(1024)])
        return {"auto": float(torch.quantile(knn, 0.95)), "radius": float(far.min())}
    if n > 25_000:
        return None
    out = {"h0": _h0(points, state["t"])}
    for k in range(1, case["max_dim"] + 1):
        h1 = _h1(points, state["t"]) if k == 1 else None  # H2 has no short way
        out["h%d" % k] = None if h1 is None else _collect([h1], state["rows"][k].double())
        out["count%d" % k] = None
    return out
