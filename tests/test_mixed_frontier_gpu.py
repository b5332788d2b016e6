"""The mixed form's per-source push against its definition restated in numpy: a round takes the whole
frontier's residuals, a vertex's sum is exact in 2^-62 fixed point, divided (rounding down) by its
degree and rounded to FP32, and every vertex that a frontier vertex reaches is in the next frontier,
also where its residual has rounded to 0.  On a grid the far vertices' residuals do after 31 rounds.
Work counters are equal."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(rows, cols):
    i = np.arange(rows * cols).reshape(rows, cols)
    u = np.concatenate([i[:, :-1].ravel(), i[:-1].ravel()])
    v = np.concatenate([i[:, 1:].ravel(), i[1:].ravel()])
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(rows * cols + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=rows * cols))
    return idx, dst[order].astype(np.uint32)


def _pushes(idx, adj, taus, eps):
    """(rounds, frontier vertices, traversals) over all sources, and how many frontier vertices had
    residual 0.  Sums stay below 4 here (4 neighbours), so 64 bits hold them."""
    idx, adj = idx.astype(np.int64), adj.astype(np.int64)
    n, m = len(idx) - 1, len(adj)
    deg = np.diff(idx)
    logmd = np.log(m / (1.0 / n))
    total = np.zeros(4, np.int64)
    for s in range(n):
        ds, tau = deg[s], taus[idx[s]:idx[s + 1]]
        r, front = np.zeros(n, np.float32), np.array([s])
        r[s] = 1.0
        ell = 0
        while True:
            total += (0, len(front), deg[front].sum(), (r[front] == 0).sum())
            sums, reached = np.zeros(n, np.uint64), np.zeros(n, bool)
            at = np.concatenate([np.arange(idx[v], idx[v + 1]) for v in front])
            fixed = np.rint(r[front].astype(np.float64) * 2.0**62).astype(np.uint64)
            np.add.at(sums, adj[at], np.repeat(fixed, deg[front]))
            reached[adj[at]] = True
            r = (sums // deg.astype(np.uint64)).astype(np.float32) * np.float32(2.0**-62)
            front = np.flatnonzero(reached)
            ell += 1
            gmax = float(r[front].max())
            gmin = 0.0 if len(front) < n else float(r[front].min())
            rest = (tau - ell)[tau > ell].astype(np.float64)
            chi = 2.0 * rest * (gmax - gmin)
            dse = float(ds) * eps
            rw = np.maximum(np.ceil(8.0 * (chi * chi) * logmd / (dse * dse)), 1.0).sum()
            if deg[front].sum() >= 25.0 * rw:
                break
        total[0] += ell
    return total


@pytest.mark.parametrize("tier", ["smem", "global"])
def test_frontier_keeps_the_vertices_whose_residual_rounded_to_zero(cuda_device, monkeypatch, tier):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_MIXED, VEC_F32

    idx, adj = _grid(12, 60)
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.98, 0.88, 15)])
    vec = np.random.default_rng(5).normal(size=n * 16).astype(np.float32)
    g = AESCGraph.from_csr(idx, adj, values, vec, VEC_F32)
    monkeypatch.setenv("TGTP_MIXED_BLOCK", "0")
    monkeypatch.setenv("TGTP_PVEC_TIER", tier)
    a = AESC(g, AESCConfig(0.05, omega=16, gamma=10, precision=PRECISION_MIXED))
    a.tgtp()
    st = a.stats()
    rounds, vertices, traversals, zeros = _pushes(idx, adj, a.taus(), 0.05)
    assert zeros > 100  # the case is there
    assert (st["push_rounds"], st["push_vertices"], st["push_traversals"]) == (rounds, vertices, traversals)
    g.free()
