"""The mixed form's per-source stage restated in numpy, for every source of small graphs: the push
(exact sums in 2^-62 fixed point, 64 bits wide), the edge bound of the top-gamma residuals, chi and the walk
count of every walking slot.  Walk counts per slot and rounds per row are equal, in shared memory, in HBM with the bitmap
of touched vertices in shared memory and in HBM, and after both block pushes; gamma up to beyond the frontier; 128 and
256 threads per block."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _graph(name):
    rng = np.random.default_rng(29)
    if name == "triangles":  # hubs of 300 neighbours, and triangles
        n = 611
        ring = np.arange(n)
        u = np.concatenate([ring, ring, np.repeat(np.array([0, 200, 400]), 300)])
        v = np.concatenate([(ring + 1) % n, (ring + 2) % n, rng.integers(0, n, 900)])
    else:  # "n3503": the size of 256 threads per block in shared memory
        n = 3503
        ring = np.arange(n)
        u = np.concatenate([ring, rng.integers(0, n, 6 * n)])
        v = np.concatenate([(ring + 1) % n, rng.integers(0, n, 6 * n)])
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


def _push(s, idx, adj, deg, tau, eps, logmd):
    """(rounds, residuals, frontier, gmax, gmin) of source s (see test_mixed_frontier_gpu.py)."""
    n, ds = len(deg), deg[s]
    r, front, ell = np.zeros(n, F), np.array([s]), 0
    r[s] = 1.0
    while True:
        at = np.concatenate([np.arange(idx[v], idx[v + 1]) for v in front])
        sums = np.zeros(n, np.uint64)
        np.add.at(sums, adj[at], np.repeat(np.rint(r[front].astype(np.float64) * 2.0**62).astype(np.uint64), deg[front]))
        r = (sums // deg.astype(np.uint64)).astype(F) * F(2.0**-62)
        front = np.unique(adj[at])
        ell += 1
        gmax, gmin = r[front].max(), F(0) if len(front) < n else r[front].min()
        rest = (tau - ell)[tau > ell].astype(np.float64)
        chi = 2.0 * rest * (float(gmax) - float(gmin))
        dse = float(ds) * eps
        rw = np.maximum(np.ceil(8.0 * (chi * chi) * logmd / (dse * dse)), 1.0).sum()
        if deg[front].sum() >= 25.0 * rw:
            return ell, r, front, gmax, gmin


def _walks(s, idx, adj, deg, tau, eps, logmd, gammas):
    """Rounds of source s, and for each gamma the walk counts of its row."""
    ell, r, front, gmax, gmin = _push(s, idx, adj, deg, tau, eps, logmd)
    row = adj[idx[s]:idx[s + 1]]
    walking = np.flatnonzero(tau > ell)
    out = {}
    if walking.size == 0:
        return ell, {g: np.zeros(len(row), np.int64) for g in gammas}
    smax, smin = r[row].max(), r[row].min()
    near = [r[adj[idx[row[k]]:idx[row[k] + 1]]] for k in walking]
    tmax, tmin = np.array([x.max() for x in near]), np.array([x.min() for x in near])
    order = front[np.argsort(-r[front], kind="stable")]
    # pairs of adjacent frontier vertices: the rank of the later one and the sum, best sum by rank
    rank = np.full(len(deg), len(order))
    rank[order] = np.arange(len(order))
    best = np.zeros(len(order) + 1, F)
    for v in order:
        nb = adj[idx[v]:idx[v + 1]]
        nb = nb[rank[nb] < rank[v]]
        if nb.size:
            best[rank[v]] = (r[v] + r[nb]).max()
    best = np.maximum.accumulate(best)
    L = (tau[walking] - ell).astype(np.int64)
    dse = F(float(deg[s]) * eps)
    for g in gammas:
        if g == 1:
            edge = F(2) * gmax
        else:
            k = min(g, len(order))
            t = F(0) if g >= len(order) else r[order[g - 1]]
            edge = max(gmax + min(F(1), t), best[k - 1])
        a = float(gmax) + (smax + tmax).astype(np.float64) / 2.0
        b = a + ((L - 1).astype(F) * edge).astype(np.float64)
        c = (b - float(smin)) - tmin.astype(np.float64)
        chi = (c - ((2 * (L - 1)).astype(F) * gmin).astype(np.float64)).astype(F)
        num = (F(8) * (chi * chi)).astype(np.float64) * logmd
        nr = np.maximum(np.ceil(num / float(dse * dse)), 1.0).astype(np.int64)
        out[g] = np.zeros(len(row), np.int64)
        out[g][walking] = nr + 8 - nr % 8
    return ell, out


@pytest.mark.parametrize("name,eps,gammas", [("triangles", 0.05, (1, 10, 64, 65, 200, 1000)), ("n3503", 0.05, (10, 300))])
def test_walk_counts_and_rounds_of_every_source(cuda_device, monkeypatch, name, eps, gammas):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_MIXED, VEC_F32

    idx, adj = _graph(name)
    n, m = len(idx) - 1, len(adj)
    values = np.concatenate([[1.0], np.linspace(0.9, 0.6, 15)])
    vec = np.random.default_rng(5).normal(size=(n, 16)) * np.random.default_rng(6).uniform(0, 1.0, size=(n, 1))
    g = AESCGraph.from_csr(idx, adj, values, vec.reshape(-1).astype(np.float32), VEC_F32)
    g.set_trace(True)
    got = {}
    for gamma in gammas:
        for path, env in (("shared", {"TGTP_MIXED_BLOCK": "0"}),
                          ("hbm", {"TGTP_MIXED_BLOCK": "0", "TGTP_PVEC_TIER": "global"}),
                          ("hbm_bits", {"TGTP_MIXED_BLOCK": "0", "TGTP_PVEC_TIER": "global", "TGTP_BLOCK_MASKS": "global"}),
                          ("block", {"TGTP_MIXED_BLOCK": "1"}),
                          ("block32", {"TGTP_MIXED_BLOCK": "1", "TGTP_BLOCK_CTAS": "148"})):
            for k in ("TGTP_MIXED_BLOCK", "TGTP_PVEC_TIER", "TGTP_BLOCK_MASKS", "TGTP_BLOCK_CTAS"):
                monkeypatch.delenv(k, raising=False)
            for k, v in env.items():
                monkeypatch.setenv(k, v)
            a = AESC(g, AESCConfig(eps, omega=16, gamma=gamma, precision=PRECISION_MIXED))
            scores = a.tgtp()
            got[gamma, path] = (scores, *g.read_trace())
            for x, y in zip(got[gamma, path], got[gamma, "shared"]):
                assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (gamma, path)
    taus = a.taus()
    g.free()
    idx, adj = idx.astype(np.int64), adj.astype(np.int64)
    deg = np.diff(idx)
    logmd = math.log(m / (1.0 / n))
    listed = [s for s in range(n) if taus[idx[s]:idx[s + 1]].max() > 1]
    some = listed if len(listed) < 700 else listed[::len(listed) // 400]
    walked = 0
    for s in some:
        ell, want = _walks(s, idx, adj, deg, taus[idx[s]:idx[s + 1]], eps, logmd, gammas)
        for gamma in gammas:
            _, nr, rounds = got[gamma, "shared"]
            assert rounds[s] == ell, (s, gamma)
            assert np.array_equal(nr[idx[s]:idx[s + 1]], want[gamma]), (s, gamma)
        walked += int((want[gammas[0]] > 0).sum())
    assert walked > 300
