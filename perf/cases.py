"""The performance cases of this framework: what a user has it do, through its public entry points.

Every case is one pass through the C ABI of libtsne_h2pack.so (include/tsne_h2pack.h) as the
package binds it, or through the Python classes over it (TSNE, the k-NN methods,
EmbeddingServer). The sizes span the benchmark's (1,000,000 points in 2D), the configurations
of the documents and tests (10K, 20K, 100K, 200K; 3D at 100K) and the smallest that each path
takes.

Kinds of pass:
  optimise  tsne_set_embedding, tsne_run_range over 60 iterations, tsne_get_embedding: the
            optimisation phase from a warm start, on a workspace that keeps P. 'late' is the
            schedule after exaggeration (H2 rebuild every third iteration), 'early' the
            exaggeration phase (every tenth), 'exact' the O(N^2) method of small inputs.
  force     tsne_set_embedding, update_h2_matrix, compute_repulsive_forces_h2pack: one H2
            build and one product.
  knn       knn_method='cuda': the exact neighbour graph of a feature matrix.
  jointp    tsne_joint_P_from_knn_distances: calibrated, symmetric P from a neighbour graph.
  fit       TSNE.fit_transform(X): neighbour graph, P, PCA start and every iteration.
  batch     EmbeddingServer: several small embeddings at once.

The embeddings are drawn, not run: clusters of Zipf(1.1) sizes with the extent, the density, the
outliers and the tight clumps that runs of the benchmark's mixture show at iteration 300-500
('late': rms 21 whatever the number of points) and 50-250 ('early': dense cores, rms 3-4, a
long tail). The neighbour graphs put each point's neighbours at log-normal distances along the
embedding's tree order (median 0.5% of the points, as those runs show), a part of them on
hubs, so rows of P differ in length as they do in 50 dimensions.
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "tsne-h2pack-python_b200"))

from tsne_h2pack import TSNE  # noqa: E402
from tsne_h2pack._backend import DTYPE, get_backend  # noqa: E402
from tsne_h2pack._knn_methods import get_knn_method  # noqa: E402
from tsne_h2pack.serving import EmbeddingServer  # noqa: E402

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
NEIGHBOURS = 90          # perplexity 30, three times as many neighbours
PERPLEXITY = 30.0
ITERS = 60


# ---------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------
def _optimise(name, n, d, phase="late", tol=None, leaf=100, freq=3):
    c = {"kind": "optimise", "n": n, "d": d, "phase": phase, "tol": tol or (1e-2 if d == 2 else 3e-2), "leaf": leaf,
         "freq": freq, "iters": ITERS}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the benchmark's size: a million cells in 2D, late in the run
        _optimise("late2d_1m", 1_000_000, 2),
        # an ordinary large data set
        _optimise("late2d_200k", 200_000, 2),
        # an ordinary small one, and the smallest that takes the H2 path: latency and launches
        _optimise("late2d_20k", 20_011, 2),
        _optimise("late2d_2k", 2_101, 2),
        # the exaggeration phase (a quarter of every run): few rebuilds, concentrated embedding
        _optimise("early2d_300k", 300_007, 2, phase="early"),
        # three dimensions at the default tolerance
        _optimise("late3d_100k", 100_003, 3),
        # method='exact', and every input below 2000 points
        _optimise("exact2d_1500", 1_501, 2, phase="exact"),
        # one H2 build and product by itself
        {"name": "force3d_20k", "kind": "force", "n": 20_000, "d": 3, "tol": 3e-2, "leaf": 100},
        # the neighbour graph of a feature matrix
        {"name": "knn_100k", "kind": "knn", "n": 100_000, "dim": 50, "k": 90},
        # P from a neighbour graph of any source
        {"name": "jointp_100k", "kind": "jointp", "n": 100_000, "d": 2},
        # the whole call on a feature matrix of ordinary size
        {"name": "fit_10k", "kind": "fit", "n": 10_000, "dim": 50, "d": 2, "iters": 1000},
        # many small embeddings served at once
        {"name": "batch_8x5k", "kind": "batch", "jobs": 8, "n": 5_000, "d": 2, "iters": 250},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["late2d"] * 5 + ["late3d"] * 3 + ["early", "early", "exact", "exact", "force", "force", "knn",
                                                            "knn", "jointp", "fit", "batch"])
    if kind == "late2d":
        return _optimise(None, _log_uniform(rng, 2_000, 600_000), 2, tol=rng.choice([1e-2, 1e-2, 3e-2, 3e-3]),
                         leaf=rng.choice([100, 100, 48, 64, 128, 160]), freq=rng.choice([3, 3, 1, 5, 10]))
    if kind == "late3d":
        return _optimise(None, _log_uniform(rng, 2_000, 90_000), 3, tol=rng.choice([3e-2, 3e-2, 1e-2]),
                         leaf=rng.choice([100, 100, 64, 160]), freq=rng.choice([3, 3, 5]))
    if kind == "early":
        return _optimise(None, _log_uniform(rng, 3_000, 600_000), rng.choice([2, 2, 3]), phase="early")
    if kind == "exact":
        return _optimise(None, _log_uniform(rng, 120, 6_000), rng.choice([2, 2, 3]), phase="exact")
    if kind == "force":
        d = rng.choice([2, 3])
        return {"kind": "force", "n": _log_uniform(rng, 2_000, 60_000), "d": d, "tol": rng.choice([1e-2, 3e-2]),
                "leaf": rng.choice([100, 64, 128])}
    if kind == "knn":
        return {"kind": "knn", "n": _log_uniform(rng, 1_000, 120_000), "dim": rng.choice([2, 10, 33, 50, 64, 90]),
                "k": rng.choice([15, 45, 90, 120])}
    if kind == "jointp":
        return {"kind": "jointp", "n": _log_uniform(rng, 1_000, 150_000), "d": 2}
    if kind == "fit":
        return {"kind": "fit", "n": _log_uniform(rng, 300, 12_000), "dim": rng.choice([20, 50]),
                "d": rng.choice([2, 2, 3]), "iters": rng.choice([300, 500])}
    return {"kind": "batch", "jobs": rng.choice([4, 6, 8]), "n": _log_uniform(rng, 1_000, 8_000),
            "d": rng.choice([2, 2, 3]), "iters": rng.choice([150, 250])}


# ---------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------
def _clusters(n, g):
    """Zipf(1.1) cluster weights and a cluster for every point."""
    k = min(100, max(5, n // 2000))
    w = torch.arange(1, k + 1, dtype=torch.float64, device=DEVICE) ** -1.1
    w = w / w.sum()
    return w, torch.multinomial(w, n, replacement=True, generator=g)


def _ball(m, d, g):
    x = torch.randn(m, d, dtype=torch.float64, device=DEVICE, generator=g)
    r = torch.rand(m, 1, dtype=torch.float64, device=DEVICE, generator=g) ** (1.0 / d)
    return x / x.norm(dim=1, keepdim=True) * r


def _embedding(n, d, phase, g):
    """(n, d) embedding, values representable in single precision."""
    w, lab = _clusters(n, g)
    early = phase == "early"
    radius = 4.0 if early else 36.0
    centre = radius * _ball(len(w), d, g)
    size = radius * (0.05 if early else 0.9) * w[lab, None] ** (1.0 / d)
    off = size * _ball(n, d, g)
    u = torch.rand(n, 1, dtype=torch.float64, device=DEVICE, generator=g)
    if early:
        off = off * u.clamp_min(3e-4) ** -1.0                    # dense cores with a long tail
    else:
        off = torch.where(u < 0.003, 1e-3 * off, off)            # a tight clump in each cluster
    y = centre[lab] + off
    if not early:
        y = torch.where(u > 0.999, y * (1.0 + 5000.0 * (u - 0.999)), y)   # a few outliers
    return (y - y.mean(0)).float().double()


def _tree_order(y):
    """The points' order along a Morton curve of the embedding."""
    lo, hi = y.min(0).values, y.max(0).values
    q = ((y - lo) / (hi - lo).max() * (2 ** 20 - 1)).long()
    key = torch.zeros(len(y), dtype=torch.long, device=y.device)
    for b in range(20):
        for k in range(y.shape[1]):
            key |= ((q[:, k] >> b) & 1) << (b * y.shape[1] + k)
    return torch.sort(key, stable=True).indices


def _graph(y, g, k=NEIGHBOURS):
    """A neighbour graph of the points (CSR of distances on the host: indptr, indices, data;
    rows sorted by column, no self entries), local in the embedding's tree order."""
    n = len(y)
    k = min(k, n - 1)
    order = _tree_order(y)
    median, sigma = max(3.0, 0.005 * n), 2.5
    cols, dist, counts = [], [], []
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device=DEVICE)
    step = 200_000
    for a in range(0, n, step):
        m = min(step, n - a)
        delta = torch.exp(sigma * torch.randn(m, k, device=DEVICE, generator=g)) * median
        delta = delta.clamp(1.0, n / 2).round().long()
        sign = torch.randint(0, 2, (m, k), device=DEVICE, generator=g) * 2 - 1
        pos = (rank[a:a + m, None] + sign * delta) % n
        hub = torch.rand(m, k, device=DEVICE, generator=g)
        pos = torch.where(hub < 0.12, pos // 16 * 16, torch.where(hub < 0.14, pos // 512 * 512, pos))
        col = torch.sort(order[pos], dim=1).values
        keep = col != torch.arange(a, a + m, device=DEVICE)[:, None]
        keep[:, 1:] &= col[:, 1:] != col[:, :-1]
        scale = 3.0 + 5.0 * torch.rand(m, 1, dtype=torch.float64, device=DEVICE, generator=g)
        far = torch.rand(m, k, dtype=torch.float64, device=DEVICE, generator=g) ** 0.25
        cols.append(col[keep].int().cpu().numpy())
        dist.append((scale * (0.75 + 0.25 * far))[keep].cpu().numpy())
        counts.append(keep.sum(1).cpu().numpy())
    ptr = np.concatenate([[0], np.cumsum(np.concatenate(counts))]).astype(np.int32)
    return ptr, np.concatenate(cols), np.concatenate(dist)


def _features(n, dim, g):
    """A Gaussian mixture of Zipf-sized clusters (float32, on the host): the benchmark's data."""
    w, lab = _clusters(n, g)
    centre = 3.0 * torch.randn(len(w), dim, device=DEVICE, generator=g)
    sd = 0.5 + 1.5 * torch.rand(len(w), dim, device=DEVICE, generator=g)
    x = centre[lab] + sd[lab] * torch.randn(n, dim, device=DEVICE, generator=g)
    return x.cpu().numpy()


def _ptr(a, t):
    return a.ctypes.data_as(ctypes.POINTER(t))


class _Workspace:
    """A workspace of the C ABI, as a program that optimises from warm starts keeps it."""

    def __init__(self, case, y0, graph):
        self.lib = get_backend()._lib
        self.n, self.d = case["n"], case["d"]
        p = get_backend().create_default_params()
        p.n_iter, p.verbose, p.perplexity = 1000, 0, min(PERPLEXITY, (self.n - 1) / 3.0)
        p.learning_rate = max(self.n / 12.0, 200.0)
        exact = case.get("phase") == "exact"
        p.h2_tol = 1e-4 if exact else case["tol"]
        p.h2_leaf_size = case["leaf"]
        p.h2_rebuild_freq = 999999 if exact else case.get("freq", 3)
        p.h2_rebuild_freq_early = max(10, p.h2_rebuild_freq)
        p.init_method, p.init_Y = 1, _ptr(y0, DTYPE)
        indptr, indices, data = graph
        self.ws = self.lib.tsne_init_with_knn_distances(None, self.n, 0, self.d, ctypes.byref(p), _ptr(data, DTYPE),
                                                        _ptr(indices, ctypes.c_int), _ptr(indptr, ctypes.c_int),
                                                        len(data))
        if not self.ws:
            raise RuntimeError("tsne_init_with_knn_distances failed")

    def __del__(self):
        if getattr(self, "ws", None):
            self.lib.tsne_destroy(self.ws)
            self.ws = None


def _inputs(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("optimise", "force"):
        phase = "early" if case.get("phase") == "early" else "late"
        y = _embedding(case["n"], case["d"], phase, g)
        # the force does not read P: a short graph stands in for it
        return {"y0": np.ascontiguousarray(y.T.cpu().numpy()),
                "graph": _graph(y, g, NEIGHBOURS if kind == "optimise" else 12)}
    if kind == "jointp":
        # which points are neighbours is the same for every seed, so that P has as many entries
        # for each; the distances, and so every value of P, are the seed's
        h = torch.Generator(device=DEVICE).manual_seed(case["n"])
        indptr, indices, data = _graph(_embedding(case["n"], case["d"], "late", h), h)
        far = torch.rand(len(data), dtype=torch.float64, device=DEVICE, generator=g).cpu().numpy()
        return {"graph": (indptr, indices, data * (0.95 + 0.05 * far))}
    if kind == "batch":
        return {"x": [_features(case["n"] + 37 * j, 20, g) for j in range(case["jobs"])]}
    return {"x": _features(case["n"], case["dim"], g)}


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("optimise", "force"):
        s["ws"] = _Workspace(case, s["y0"], s["graph"])
        if kind == "force":
            lib = s["ws"].lib
            lib.update_h2_matrix.argtypes = [type(s["ws"].ws), ctypes.c_int]
            lib.tsne_get_h2_matrix.argtypes = [type(s["ws"].ws)]
            lib.tsne_get_h2_matrix.restype = ctypes.c_void_p
            lib.compute_repulsive_forces_h2pack.argtypes = [ctypes.c_void_p, ctypes.POINTER(DTYPE), ctypes.c_int,
                                                            ctypes.c_int, type(s["ws"].ws), ctypes.POINTER(DTYPE),
                                                            ctypes.c_int]
            lib.compute_repulsive_forces_h2pack.restype = ctypes.c_double
    elif kind == "batch":
        # a serving process keeps its server; the jobs' probabilities come with the requests
        be, knn = get_backend(), get_knn_method("cuda")
        s["P"] = [be.joint_P_device(knn.compute(x, k=NEIGHBOURS), PERPLEXITY) for x in s["x"]]
        s["server"] = EmbeddingServer(max_concurrent=case["jobs"], hbm_budget_gb=100.0)
    return s


# ---------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------
def _begin(case):
    """First iteration of the pass, a rebuild iteration of its schedule."""
    return 110 if case["phase"] == "early" else 300


def _run_optimise(s):
    c, w = s["case"], s["ws"]
    if w.lib.tsne_set_embedding(w.ws, s["y0"]) != 0:
        raise RuntimeError("tsne_set_embedding failed")
    if w.lib.tsne_run_range(w.ws, _begin(c), _begin(c) + c["iters"]) != 0:
        raise RuntimeError("tsne_run_range failed")
    y = np.empty((c["d"], c["n"]))
    w.lib.tsne_get_embedding(w.ws, y)
    return {"embedding": y.astype(np.float32)}   # the engine's state is single precision


def _run_force(s):
    c, w = s["case"], s["ws"]
    if w.lib.tsne_set_embedding(w.ws, s["y0"]) != 0 or w.lib.update_h2_matrix(w.ws, 1) != 0:
        raise RuntimeError("update_h2_matrix failed")
    grad = np.zeros((c["d"], c["n"]))
    h = w.lib.tsne_get_h2_matrix(w.ws)
    z = w.lib.compute_repulsive_forces_h2pack(h, _ptr(s["y0"], DTYPE), c["d"], c["n"], w.ws, _ptr(grad, DTYPE), 0)
    return {"grad": grad.astype(np.float32), "Z": np.float32(z)}   # computed in single precision


def _run_knn(s):
    G = get_knn_method("cuda").compute(s["x"], k=s["case"]["k"])
    return {"indices": G.indices, "distances": G.data.astype(np.float32)}


def _run_jointp(s):
    indptr, indices, data = s["graph"]
    lib, n = get_backend()._lib, s["case"]["n"]
    m = lib.tsne_joint_P_from_knn_distances(_ptr(data, DTYPE), _ptr(indices, ctypes.c_int), _ptr(indptr, ctypes.c_int),
                                            n, len(data), PERPLEXITY)
    if not m:
        raise RuntimeError("tsne_joint_P_from_knn_distances failed")
    c = m.contents
    out = {"row_ptr": np.ctypeslib.as_array(c.row_ptr, shape=(n + 1,)).copy(),
           "col_idx": np.ctypeslib.as_array(c.col_idx, shape=(c.nnz,)).copy(),
           "values": np.ctypeslib.as_array(c.values, shape=(c.nnz,)).copy()}
    lib.sparse_matrix_destroy(m)
    return out


def _run_fit(s):
    c = s["case"]
    est = TSNE(n_components=c["d"], perplexity=min(PERPLEXITY, (c["n"] - 1) / 3.0), max_iter=c["iters"],
               random_state=1, knn_method="cuda")
    return {"embedding": est.fit_transform(s["x"]).astype(np.float32)}


def _run_batch(s):
    c = s["case"]
    rate = [max(P.shape[0] / 12.0, 200.0) for P in s["P"]]
    jobs = [s["server"].submit(P, n_components=c["d"], n_iter=c["iters"], verbose=0, learning_rate=r, random_seed=j,
                               h2_tol=1e-2 if c["d"] == 2 else 3e-2, h2_rebuild_freq=3, h2_rebuild_freq_early=10)
            for j, (P, r) in enumerate(zip(s["P"], rate))]
    out = []
    for j in jobs:
        y, info = s["server"].wait(j)
        if not info.ok:
            raise RuntimeError("a served job failed")
        out.append(y.astype(np.float32))
    return {"embeddings": out}


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------
def work(case):
    """Inputs read once per use and outputs written once. An optimise pass reads P and the
    points' state in every iteration; its repulsion is counted at the 600 kernel evaluations
    per point that an H2 product of these tolerances needs at each rebuild."""
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("optimise", "fit", "batch"):
        d, its = case["d"], case["iters"]
        nnz = 160.0 * n
        nb = max(1, its // 3) if kind != "optimise" else its // (10 if case["phase"] == "early" else case["freq"])
        pairs = its * float(n) * n if case.get("phase") == "exact" or n < 2000 else nb * 600.0 * n
        reps = case.get("jobs", 1)
        return {"bytes": reps * (its * (8.0 * nnz + 4.0 * n + 28.0 * d * n) + 16.0 * d * n),
                "flops": reps * (its * nnz + pairs) * (3 * d + 5)}
    if kind == "force":
        d = case["d"]
        return {"bytes": 16.0 * d * n, "flops": 600.0 * n * (3 * d + 5)}
    if kind == "knn":
        return {"bytes": 4.0 * n * case["dim"] + 8.0 * n * case["k"], "flops": 2.0 * case["dim"] * n * n}
    return {"bytes": 12.0 * NEIGHBOURS * n + 12.0 * 160 * n, "flops": 40.0 * NEIGHBOURS * n}


# ---------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------
def _exact_repulsion(y, step=2_000):
    """(F, Z): F_i = 4/Z sum_j (y_i - y_j) / (1 + r^2)^2, Z = sum_{i != j} 1 / (1 + r^2)."""
    force, z = torch.empty_like(y), torch.zeros((), dtype=torch.float64, device=y.device)
    for a in range(0, len(y), step):
        b = y[a:a + step]
        w = torch.ones(len(b), len(y), dtype=torch.float64, device=y.device)
        for k in range(y.shape[1]):
            w += (b[:, k, None] - y[None, :, k]) ** 2
        w.reciprocal_()
        z += w.sum() - len(b)
        w.mul_(w)
        force[a:a + step] = b * w.sum(1, keepdim=True) - w @ y
    return 4.0 / z * force, z


def _exact_joint_p(n, graph, perplexity):
    """(row, col, value) of P: beta by bisection to 1e-5 of the entropy, then (P + P^T) / sum."""
    indptr, indices, data = (torch.as_tensor(a, device=DEVICE) for a in graph)
    count = (indptr[1:] - indptr[:-1]).long()
    width = int(count.max())
    row = torch.repeat_interleave(torch.arange(n, device=DEVICE), count)
    at = torch.arange(len(data), device=DEVICE) - indptr.long()[row]
    d2 = torch.full((n, width), math.inf, dtype=torch.float64, device=DEVICE)
    d2[row, at] = data * data
    d2 = d2 - d2.min(1, keepdim=True).values
    live, d2 = torch.isfinite(d2), torch.nan_to_num(d2, posinf=0.0)
    beta = torch.ones(n, dtype=torch.float64, device=DEVICE)
    lo, hi, done = torch.zeros_like(beta), torch.full_like(beta, math.inf), torch.zeros(n, dtype=torch.bool, device=DEVICE)
    for _ in range(200):
        p = torch.exp(-beta[:, None] * d2) * live
        total = p.sum(1)
        diff = torch.log(total) + beta * (d2 * p).sum(1) / total - math.log(perplexity)
        done = done | (diff.abs() < 1e-5)
        if bool(done.all()):
            break
        up = ~done & (diff > 0)
        down = ~done & (diff <= 0)
        lo, hi = torch.where(up, beta, lo), torch.where(down, beta, hi)
        nxt = torch.where(up, torch.where(torch.isinf(hi), 2 * beta, 0.5 * (beta + hi)),
                          torch.where(lo == 0, 0.5 * beta, 0.5 * (beta + lo)))
        beta = torch.where(done, beta, nxt)
    p = (p / total[:, None])[row, at]
    col = indices.long()
    key, inverse = torch.unique(torch.cat([row * n + col, col * n + row]), return_inverse=True)
    value = torch.zeros(len(key), dtype=torch.float64, device=DEVICE).index_add_(0, inverse, torch.cat([p, p]))
    key, value = key[value != 0], value[value != 0]
    return key // n, key % n, value / value.sum()


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "force" and n <= 60_000:
        f, z = _exact_repulsion(torch.as_tensor(_inputs(case, seed)["y0"].T.copy(), device=DEVICE))
        return {"grad": -f.T.cpu().numpy(), "Z": z.cpu().numpy()}
    if kind == "jointp":
        row, col, value = _exact_joint_p(n, _inputs(case, seed)["graph"], PERPLEXITY)
        return {"row_ptr": None, "col_idx": None, "values": value.cpu().numpy()}
    if kind == "knn":
        x = torch.as_tensor(_inputs(case, seed)["x"], device=DEVICE).double()
        out = []
        for a in range(0, n, 500):
            d2 = torch.cdist(x[a:a + 500], x, compute_mode="donot_use_mm_for_euclid_dist")
            d2[torch.arange(len(d2)), torch.arange(a, a + len(d2))] = math.inf
            v, i = torch.topk(d2, case["k"], dim=1, largest=False)
            out.append(torch.gather(v, 1, torch.sort(i, dim=1).indices))
        return {"indices": None, "distances": torch.cat(out).reshape(-1).cpu().numpy()}
    if kind == "optimise" and case["phase"] == "exact":
        s = _inputs(case, seed)
        row, col, p = _exact_joint_p(n, s["graph"], min(PERPLEXITY, (n - 1) / 3.0))
        y = torch.as_tensor(s["y0"].T.copy(), device=DEVICE)
        u, gain, rate = torch.zeros_like(y), torch.ones_like(y), max(n / 12.0, 200.0)
        P = torch.zeros(n, n, dtype=torch.float64, device=DEVICE)
        P[row, col] = p
        for _ in range(case["iters"]):
            w = torch.ones(n, n, dtype=torch.float64, device=DEVICE)
            for k in range(y.shape[1]):
                w += (y[:, k, None] - y[None, :, k]) ** 2
            w = P / w
            g = 4.0 * (y * w.sum(1, keepdim=True) - w @ y) - _exact_repulsion(y)[0]
            gain = torch.where(u * g < 0, gain + 0.2, gain * 0.8).clamp_min(0.01)
            u = 0.8 * u - rate * gain * g
            y = y + u
            y = y - y.mean(0)
        return {"embedding": y.T.cpu().numpy()}
    # An H2 run over many iterations amplifies every rounding (about 1e-3 after 30 iterations at
    # 200,000 points, and more from a random start): no 64-bit value says what it should return.
    return None
