"""The work that users of this framework have it do, as cases that can be timed and compared.

Three kinds of call carry the framework, and every case is one of them through its public entry
points (tgtp_b200.aesc):

* scores     tgtp() on a graph that is resident on the device (`AESC.tgtp_device`), the whole call
             with host data as the command-line runner makes it (`AESCGraph.from_csr`,
             `upload_eigens`, `AESC.tgtp`), and many graphs as one batch (`Batch`);
* walks      the SABA walk counter (`saba_count`) and the MT19937 comparison walks
             (`mt_walk_count`);
* accuracy   the exact spanning centrality of sampled edges (`exact_sc_slots`), against which the
             scores' error is stated.

Graphs are the repository's three kinds of synthetic graph (Chung-Lu power law, R-MAT, 2-D grid with
random chords; connected, no self-loops, sorted CSR), drawn on the GPU from the seed with the case's
numbers of vertices and edges.
omega = 128 eigenpairs of the normalised adjacency matrix, the largest |lambda| first, come from a
few rounds of Chebyshev-filtered subspace iteration (residuals below 1e-4); they are rounded to 24 bits so that every
storage type holds the same numbers.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from tgtp_b200 import aesc as A

_FORMS = {"fp32": A.PRECISION_FP32, "fp64": A.PRECISION_FP64, "mixed": A.PRECISION_MIXED}
_STORES = {"f32": A.VEC_F32, "f64": A.VEC_F64, "bf16": A.VEC_BF16}


# ---- graphs -------------------------------------------------------------------------------------


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _distinct(n: int, a, b):
    """Keys lo * n + hi of the distinct undirected pairs, sorted; self-loops dropped."""
    keep = a != b
    a, b = a[keep], b[keep]
    return torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b))


def _components(n: int, lo, hi):
    """Component label of every vertex: the smallest vertex id in it."""
    label = torch.arange(n, device="cuda")
    while True:
        low = torch.minimum(label[lo], label[hi])
        new = label.scatter_reduce(0, label[lo], low, "amin").scatter_reduce(0, label[hi], low, "amin")
        new = new[new]
        if torch.equal(new, label):
            return label
        label = new


def _connected(n: int, key, edges: int, gen):
    """(n, CSR offsets, CSR neighbours) of a connected graph with exactly `edges` edges: the first
    of `key`, and for each smaller component they leave one edge into the largest."""
    take = edges
    while True:
        lo, hi = key[:take] // n, key[:take] % n
        label = _components(n, lo, hi)
        size = torch.bincount(label, minlength=n)
        over = take + int((size > 0).sum()) - 1 - edges
        if over <= 0:
            break
        take -= over
    big = torch.argmax(size)
    ends = lo[label[lo] == big]
    roots = torch.nonzero((size > 0) & (torch.arange(n, device="cuda") != big)).flatten()
    at = (torch.rand(roots.numel(), generator=gen, device="cuda", dtype=torch.float64) * ends.numel()).long()
    lo, hi = torch.cat([lo, ends[at]]), torch.cat([hi, roots])
    both = torch.sort(torch.cat([lo * n + hi, hi * n + lo])).values
    idx = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    idx[1:] = torch.cumsum(torch.bincount(both // n, minlength=n), 0)
    return n, idx, both % n


def _graph(c: dict, seed: int):
    """A connected simple graph with c["n"] vertices and c["edges"] edges."""
    gen = _generator(seed)
    n, edges = c["n"], c["edges"]

    def rand(k):
        return torch.rand(k, generator=gen, device="cuda", dtype=torch.float64)

    def until_enough(pairs, key):
        """Distinct pairs drawn by pairs(count), after `key`, until there are enough; new ones in
        random order."""
        new = torch.empty(0, dtype=torch.int64, device="cuda")
        while key.numel() + new.numel() < edges:
            more = pairs(int((edges - key.numel() - new.numel()) * 1.5) + 4096)
            new = torch.unique(torch.cat([new, more[~torch.isin(more, key)]]))
        return torch.cat([key, new[torch.randperm(new.numel(), generator=gen, device="cuda")]])

    none = torch.empty(0, dtype=torch.int64, device="cuda")
    if c["graph"] == "chung_lu":
        w = torch.arange(1, n + 1, device="cuda", dtype=torch.float64) ** (-1.0 / (c["exponent"] - 1.0))
        cdf = torch.cumsum(w / w.sum(), 0)

        def pairs(k):
            a, b = (torch.searchsorted(cdf, rand(k), right=True).clamp_(max=n - 1) for _ in range(2))
            return _distinct(n, a, b)

        key = until_enough(pairs, none)
    elif c["graph"] == "rmat":
        # the n ids of highest degree of an R-MAT graph (a = 0.57, b = c = 0.19); many of its
        # 2^scale ids have no edge
        wide = 1 << c["scale"]

        def quadrants(k):
            u = torch.zeros(k, dtype=torch.int64, device="cuda")
            v = torch.zeros_like(u)
            for _ in range(c["scale"]):
                r = rand(k)
                u = (u << 1) | (r >= 0.76)
                v = (v << 1) | (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
            return u, v

        first = quadrants(edges)
        deg = torch.bincount(torch.cat(first), minlength=wide)
        kept = torch.sort(torch.argsort(deg, descending=True, stable=True)[:n]).values
        new_id = torch.full((wide,), -1, device="cuda")
        new_id[kept] = torch.arange(n, device="cuda")

        def pairs(k, drawn=None):
            u, v = (new_id[x] for x in (drawn or quadrants(k)))
            keep = (u >= 0) & (v >= 0)
            return _distinct(n, u[keep], v[keep])

        key = pairs(0, first)
        key = until_enough(pairs, key[torch.randperm(key.numel(), generator=gen, device="cuda")])
    else:  # 2-D grid with random chords
        ids = torch.arange(n, device="cuda").reshape(c["rows"], c["cols"])
        key = torch.cat([(ids[:, :-1] * n + ids[:, 1:]).reshape(-1), (ids[:-1] * n + ids[1:]).reshape(-1)])
        key = until_enough(lambda k: _distinct(n, (rand(k) * n).long(), (rand(k) * n).long()), key)
    return _connected(n, key, edges, gen)


def _host_csr(idx, adj):
    return idx.cpu().numpy().astype(np.uint32), adj.cpu().numpy().astype(np.uint32)


def _eigenpairs(n: int, idx, adj, omega: int, seed: int):
    """(values[omega], vertex-major vectors (n, omega)), sorted by |lambda| descending, each vector
    scaled by sqrt(2m / deg): what sorted_eigens_<omega>.txt holds."""
    deg = (idx[1:] - idx[:-1]).double()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), idx[1:] - idx[:-1])
    torch.sparse.check_sparse_tensor_invariants.disable()
    p = torch.sparse_csr_tensor(idx, adj, 1.0 / torch.sqrt(deg[row] * deg[adj]), (n, n))
    x = torch.randn(n, min(n, omega + 24), generator=_generator(seed + 1), device="cuda", dtype=torch.float64)

    def orthonormal(x):
        for k in range(3):  # shifted Cholesky QR, then twice plain
            x = x / torch.linalg.vector_norm(x, dim=0)
            h = x.T @ x
            h.diagonal().add_(1e-11 * x.shape[1] if k == 0 else 0.0)
            r = torch.linalg.cholesky(h, upper=True)
            x = torch.linalg.solve_triangular(r, x, upper=True, left=False)
        return x

    def ritz(x):
        px = p @ x
        h = x.T @ px
        theta, w = torch.linalg.eigh(0.5 * (h + h.T))
        order = torch.argsort(theta.abs(), descending=True, stable=True)
        theta, w = theta[order], w[:, order]
        return px @ w, theta, x @ w

    x = orthonormal(x)
    for _ in range(40):
        px, theta, x = ritz(x)
        if float(torch.linalg.vector_norm(px - x * theta, dim=0)[:omega].max()) < 1e-4:
            break
        c = float(theta[-1].abs().clamp(min=1e-3))
        y0, y1 = x, px / c  # T_16(P / c): even, at most 1 on [-c, c]
        for _ in range(15):
            y0, y1 = y1, 2.0 * (p @ y1) / c - y0
            s = torch.linalg.vector_norm(y1, dim=0)
            y0, y1 = y0 / s, y1 / s
        x = orthonormal(y1)
    theta, x = theta[:omega].clamp(-1.0, 1.0), x[:, :omega]
    x = (x * torch.sqrt(deg.sum() / deg)[:, None]).float()
    return theta.float().double().cpu().numpy(), x.cpu().numpy()


# ---- the cases ----------------------------------------------------------------------------------

_CL4K = {"graph": "chung_lu", "n": 4039, "edges": 88234, "exponent": 2.5}
_SPARSE = {"graph": "chung_lu", "n": 25860, "edges": 119972, "exponent": 2.1}


def _score(form: str, eps: float, store: str | None = None, **more) -> dict:
    store = store or {"fp32": "f32", "fp64": "f64", "mixed": "f32"}[form]
    return {"kind": "score", "form": form, "store": store, "eps": eps, "omega": 128, "gamma": 10, **more}


def listed():
    return [
        # one run of the `tgtp` command in its default form, file parsing left out: host CSR and
        # eigenvectors in, scores on the host out
        {"name": "call_fp32_4k_e01", **_score("fp32", 0.01), **_CL4K, "kind": "call"},
        # the benchmark's headline: a resident graph of social-network size at a coarse accuracy,
        # where launches and latency count
        {"name": "fp64_4k_e05", **_score("fp64", 0.05), **_CL4K},
        # the same graph at the finest accuracy of the experiments: push and walks on most rows
        {"name": "fp64_4k_e005", **_score("fp64", 0.005), **_CL4K},
        {"name": "mixed_bf16_4k_e005", **_score("mixed", 0.005, "bf16"), **_CL4K},
        # a sparse graph whose residual vectors do not fit in shared memory: deep pushes
        {"name": "fp64_sparse_e05", **_score("fp64", 0.05), **_SPARSE},
        {"name": "mixed_sparse_e005", **_score("mixed", 0.005), **_SPARSE},
        # a large graph at the coarse accuracy
        {"name": "mixed_200k_e05", **_score("mixed", 0.05), "graph": "chung_lu", "n": 200_000,
         "edges": 2_000_000, "exponent": 2.3},
        # many small graphs of uneven size and accuracy, replayed as one launch
        {"name": "batch16", "kind": "batch", "form": "mixed", "store": "f32", "omega": 128,
         "gamma": 10, "graphs": 16, "low": 1000, "high": 3500},
        # the walk experiment's two graphs: one resident in L2, one at throughput scale
        {"name": "saba_4k_d5", "kind": "saba", "depth": 5, "walks": 2048, **_CL4K},
        {"name": "saba_rmat18_d10", "kind": "saba", "depth": 10, "walks": 2048, "graph": "rmat",
         "scale": 18, "n": 173_957, "edges": 3_806_923},
        # the walk experiment's comparison rows
        {"name": "mt_rmat16_d5", "kind": "mt", "depth": 5, "walks": 2048, "simd": False,
         "graph": "rmat", "scale": 16, "n": 46_703, "edges": 909_984},
        # the accuracy reference on a sample of edges
        {"name": "exact_sparse_256", "kind": "exact", "slots": 256, **_SPARSE},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(n: int, ratio: float, deg: float) -> dict:
    rows = max(8, int(math.sqrt(n) * ratio))
    cols = max(8, n // rows)
    return {"graph": "grid", "rows": rows, "cols": cols, "n": rows * cols,
            "edges": max(2 * rows * cols, int(rows * cols * deg / 2))}


def _rmat(n: int, deg: float) -> dict:
    return {"graph": "rmat", "scale": max(10, math.ceil(math.log2(n / 0.75))), "n": n, "edges": int(n * deg / 2)}


def _chung_lu(n: int, deg: float, exponent: float) -> dict:
    return {"graph": "chung_lu", "n": n, "edges": int(n * deg / 2), "exponent": round(exponent, 2)}


def _draw_graph(rng, lo: int, hi: int, deg_lo: float, deg_hi: float) -> dict:
    """One of the three kinds with lo..hi vertices."""
    n, deg = _log(rng, lo, hi), rng.uniform(deg_lo, deg_hi)
    kind = rng.choice(["chung_lu", "rmat", "grid"])
    if kind == "chung_lu":
        return _chung_lu(n, deg, rng.uniform(2.2, 2.8))
    return _rmat(n, deg) if kind == "rmat" else _grid(n, rng.uniform(0.5, 1.5), deg)


def draw(rng):
    kind = rng.choice(["call", "score", "score", "score", "large", "sparse", "batch", "saba", "saba", "mt", "exact"])
    form, store = rng.choice([("fp32", "f32"), ("fp64", "f64"), ("mixed", "f32"), ("mixed", "bf16")])
    if kind in ("call", "score"):  # graphs that fit an SM's shared memory, every accuracy
        return {**_score(form, rng.choice([0.05, 0.01, 0.005]), store), **_draw_graph(rng, 1000, 5000, 14, 46),
                "kind": kind, "omega": rng.choice([128, 128, 96, 50]), "gamma": rng.choice([10, 10, 1, 20])}
    if kind == "large":  # up to the large listed graph, at the coarse accuracy
        n = _log(rng, 20_000, 180_000)
        return {**_score(form, 0.05, store), **_chung_lu(n, rng.uniform(18, 28), rng.uniform(2.3, 2.7))}
    if kind == "sparse":  # deep pushes beyond shared memory
        n = _log(rng, 9000, 26_000)
        return {**_score(form, 0.05, store), **_chung_lu(n, rng.uniform(9, 13), rng.uniform(2.1, 2.4))}
    if kind == "batch":
        low = _log(rng, 500, 1200)
        return {"kind": "batch", "form": form, "store": store, "omega": 128, "gamma": 10,
                "graphs": rng.randint(3, 16), "low": low, "high": int(low * rng.uniform(1.5, 2.9))}
    if kind == "exact":
        return {"kind": "exact", "slots": rng.randint(1, 250), **_draw_graph(rng, 1000, 20_000, 8, 30)}
    depth = rng.randint(2, 15)
    if kind == "saba":
        g = _draw_graph(rng, 1000, 240_000, 6, 30)
        most = min(16384, 3.2e9 / (g["n"] * depth))
        return {"kind": kind, "depth": depth, "walks": 8 * max(1, _log(rng, 64, most) // 8), **g}
    g = _draw_graph(rng, 1000, 60_000, 6, 30)
    most = min(8192, 4e8 / (g["n"] * depth))
    return {"kind": kind, "depth": depth, "walks": 8 * max(1, _log(rng, 64, most) // 8),
            "simd": rng.random() < 0.5, **g}


def _batch_members(c: dict):
    """The batch's graphs: sizes log-uniform, kinds in turn, average degree 8-36, an eps each."""
    rng = random.Random(1000 * c["low"] + c["graphs"])
    for i in range(c["graphs"]):
        n, deg = _log(rng, c["low"], c["high"]), rng.uniform(8, 36)
        eps = rng.choice([0.05, 0.01, 0.005])
        if i % 3 == 0:
            g = _chung_lu(n, deg, rng.uniform(2.2, 2.8))
        else:
            g = _rmat(n, deg) if i % 3 == 1 else _grid(n, 1.0, deg)
        yield g, eps


# ---- preparing and running ----------------------------------------------------------------------

_stream = None


def _user_stream() -> int:
    """One stream for the whole program, as a program with its own stream would use it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _resident(c: dict, graph: dict, eps: float, seed: int):
    n, idx, adj = _graph(graph, seed)
    values, vectors = _eigenpairs(n, idx, adj, c["omega"], seed)
    g = A.AESCGraph.from_csr(*_host_csr(idx, adj))
    g.set_stream(_user_stream())
    g.upload_eigens(values, vectors.astype(np.float64) if c["store"] == "f64" else vectors, _STORES[c["store"]])
    return A.AESC(g, _config(c, eps))


def _config(c: dict, eps: float) -> A.AESCConfig:
    vec = _STORES[c["store"]] if c["form"] == "mixed" else A.VEC_F32
    return A.AESCConfig(eps, omega=c["omega"], gamma=c["gamma"], precision=_FORMS[c["form"]], vec_dtype=vec)


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        runs = []
        for i, (graph, eps) in enumerate(_batch_members(c)):
            a = _resident(c, graph, eps, seed * 64 + i)
            runs.append((a, torch.empty(a.g.m, dtype=torch.float32, device="cuda")))
        batch = A.Batch([(a, out.data_ptr()) for a, out in runs])
        return {**c, "batch": batch, "runs": runs}
    if c["kind"] == "score":
        a = _resident(c, c, c["eps"], seed)
        return {**c, "aesc": a, "out": torch.empty(a.g.m, dtype=torch.float32, device="cuda")}
    n, idx, adj = _graph(c, seed)
    if c["kind"] == "call":
        values, vectors = _eigenpairs(n, idx, adj, c["omega"], seed)
        vectors = vectors.astype(np.float64) if c["store"] == "f64" else vectors
        return {**c, "csr": _host_csr(idx, adj), "values": values, "vectors": vectors}
    g = A.AESCGraph.from_csr(*_host_csr(idx, adj))
    g.set_stream(_user_stream())
    if c["kind"] == "exact":
        return {**c, "g": g, "at": _sample(g.m, c["slots"], seed)}
    return {**c, "g": g}


def _sample(m: int, count: int, seed: int):
    return np.random.RandomState(seed).randint(0, m, count).astype(np.uint32)


def run(state):
    s = state
    if s["kind"] == "score":
        s["aesc"].tgtp_device(s["out"].data_ptr())
        return s["out"]
    if s["kind"] == "call":
        g = A.AESCGraph.from_csr(*s["csr"])
        g.upload_eigens(s["values"], s["vectors"], _STORES[s["store"]])
        scores = A.AESC(g, _config(s, s["eps"])).tgtp()
        g.free()
        return scores
    if s["kind"] == "batch":
        s["batch"].run(_user_stream())
        return [out for _, out in s["runs"]]
    if s["kind"] == "saba":
        return A.saba_count(s["g"], s["depth"], s["walks"])
    if s["kind"] == "mt":
        return A.mt_walk_count(s["g"], s["depth"], s["walks"], simd=s["simd"])
    resistance, _ = A.exact_sc_slots(s["g"], s["at"])
    return resistance


def work(case):
    """The CSR and eigenvectors read once and the results written once.  A score's operations are
    its eigenvector terms (a difference, a square and two weighted sums per undirected edge and
    pair); a walk's are about 12 integer operations a hop; a resistance's, one pass over the
    Laplacian.  Pushes and walks of a score depend on the data and are left out."""
    c = case
    if c["kind"] == "batch":
        members = [g for g, _ in _batch_members(c)]
        n, m = sum(g["n"] for g in members), sum(2 * g["edges"] for g in members)
    else:
        n, m = c["n"], 2 * c["edges"]
    csr = 4 * (n + 1) + 4 * m
    if c["kind"] in ("score", "call", "batch"):
        size = {"f32": 4, "f64": 8, "bf16": 2}[c["store"]]
        return {"bytes": csr + n * c["omega"] * size + 4 * m, "flops": 6.0 * c["omega"] * m / 2}
    if c["kind"] == "exact":
        return {"bytes": csr + 12 * c["slots"], "flops": 2.0 * m * c["slots"]}
    return {"bytes": csr + 4 * n, "flops": 12.0 * n * c["walks"] * c["depth"]}


# ---- what the results are in 64 bits ------------------------------------------------------------


def exact(case, seed):
    """Resistances by a dense factorisation of the Laplacian; scores where no row pushes beyond its
    first round.  Counters are whole numbers and need none; scores with deeper pushes and walks
    would take a sequential pass over every frontier of every source, far over 20 seconds."""
    c = case
    if c["kind"] == "exact":
        return _resistances(c, seed)
    if c["kind"] in ("score", "call"):
        return _first_round_scores(c, seed)
    return None


def _resistances(c: dict, seed: int):
    n, idx, adj = _graph(c, seed)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), idx[1:] - idx[:-1])
    lap = torch.full((n, n), 1.0 / n, dtype=torch.float64, device="cuda")  # L + J/n
    lap[row, adj] -= 1.0
    lap.diagonal().add_((idx[1:] - idx[:-1]).double())
    at = torch.from_numpy(_sample(adj.numel(), c["slots"], seed).astype(np.int64)).cuda()
    u, v, k = row[at], adj[at], torch.arange(c["slots"], device="cuda")
    b = torch.zeros(n, c["slots"], dtype=torch.float64, device="cuda")
    b[u, k] += 1.0
    b[v, k] -= 1.0
    x = torch.cholesky_solve(b, torch.linalg.cholesky(lap))
    return (x[u, k] - x[v, k]).cpu().numpy()


def _first_round_scores(c: dict, seed: int):
    """1/du + 1/dv - 2/(du dv) per slot (u, v) when the walk-length bound of every edge is 1."""
    n, idx, adj = _graph(c, seed)
    values, vectors = _eigenpairs(n, idx, adj, c["omega"], seed)
    lam, x = torch.from_numpy(values).cuda(), torch.from_numpy(vectors).cuda().double()
    deg = (idx[1:] - idx[:-1]).double()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), idx[1:] - idx[:-1])
    m, eps = adj.numel(), c["eps"] / 2
    inner = slice(1, c["omega"] - 1)
    for lo in range(0, m, 1 << 20):
        u, v = row[lo:lo + (1 << 20)], adj[lo:lo + (1 << 20)]
        d2 = (x[u, inner] - x[v, inner]) ** 2
        ups = (d2 * (1 + lam[inner])).sum(1) / m
        dlt = (d2 * (lam[inner] ** 2 / (1 - lam[inner]))).sum(1) / m
        z = 1 / deg[u] + 1 / deg[v] - 2 / (deg[u] * deg[v])

        def steps(z, eps, l):
            y = (z / eps / (1 - l * l)).clamp(min=1.0)
            return torch.ceil(torch.log(y) / torch.log(1 / l.abs()) - 1).clamp(min=1)

        first = steps(z, eps, lam[1])
        left = torch.where(eps - dlt > 0, eps - dlt, torch.full_like(dlt, eps))
        second = steps(z - ups, left, lam[c["omega"] - 1])
        if bool((torch.minimum(first, second) > 1).any()):
            return None
    return (1 / deg[row] + 1 / deg[adj] - 2 / (deg[row] * deg[adj])).cpu().numpy()
