"""The FP32 and FP64 forms' per-source kernel against the oracle, bit for bit (the same operations in
the same order, so no tolerance), in shared memory and in HBM, windowed and one vertex at a time,
with 128 and 64 threads per block, on graphs at the sizes where it changes path: rows around one and
four 32-entry steps, more vertices than the window filter has bits, tops of 1 to 100 values (more
than one group of maxima), repeated edges and self-loops."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTERS = ("push_rounds", "push_vertices", "push_traversals", "walk_edges", "walk_count", "walk_hops",
            "fallback_bouquets")


def _csr(n, u, v, keep_all=False):
    if not keep_all:
        key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
        u, v = key // n, key % n
        u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


def _graph(name):
    rng = np.random.default_rng(11)
    if name == "steps":  # hubs of 31 .. 33, 127 .. 129 neighbours on a ring
        n = 1201
        ring = np.arange(n)
        u, v = [ring], [(ring + 1) % n]
        for k, deg in enumerate((31, 32, 33, 127, 128, 129)):
            hub = 10 * (k + 1)
            others = rng.choice(np.arange(100, n), deg - 2, replace=False)
            u.append(np.full(len(others), hub))
            v.append(others)
        return _csr(n, np.concatenate(u), np.concatenate(v))
    if name == "heavy":  # about 120 neighbours each
        n = 517
        return _csr(n, np.repeat(np.arange(n), 60), rng.integers(0, n, 60 * n))
    if name == "multi":  # repeated edges and self-loops, kept
        n = 403
        ring = np.arange(n)
        u = np.concatenate([ring, ring, rng.integers(0, 30, n), ring[:40]])
        v = np.concatenate([(ring + 1) % n, (ring + 1) % n, rng.integers(0, n, n), ring[:40]])
        return _csr(n, u, v, keep_all=True)
    n = 9001  # "wide": hubs and a sparse rest
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, 50, n), rng.integers(0, n, n)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, n), rng.integers(0, n, n)])
    return _csr(n, u, v)


@pytest.mark.parametrize("fp64", [False, True], ids=["fp32", "fp64"])
@pytest.mark.parametrize("name,eps,gammas", [("steps", 0.02, (1, 10, 100)), ("heavy", 0.002, (1, 40, 100)),
                                             ("multi", 0.02, (1, 10, 40)), ("wide", 0.2, (10, 65))])
def test_push_variants_equal_the_oracle(cuda_device, oracle_lib, monkeypatch, name, eps, gammas, fp64):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_FP32, PRECISION_FP64, VEC_F32, VEC_F64

    idx, adj = _graph(name)
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.8, 0.5, 15)])
    vec = np.random.default_rng(5).normal(size=n * 16) / np.sqrt(n)
    vec = vec if fp64 else vec.astype(np.float32)
    g = AESCGraph.from_csr(idx, adj, values, vec, VEC_F64 if fp64 else VEC_F32)
    pushed = 0
    for gamma in gammas:
        want, det = oracle_lib.tgtp(idx, adj, values, vec, eps, gamma=gamma, fp64=fp64, details=True)
        for tier in (None, "smem", "global"):
            for window in (None, "0", "1"):
                for k, v in (("TGTP_PVEC_TIER", tier), ("TGTP_GS_WINDOW", window)):
                    if v is None:
                        monkeypatch.delenv(k, raising=False)
                    else:
                        monkeypatch.setenv(k, v)
                a = AESC(g, AESCConfig(eps, omega=16, gamma=gamma, precision=PRECISION_FP64 if fp64 else PRECISION_FP32))
                got = a.tgtp()
                st = a.stats()
                bad = np.flatnonzero(got.view(np.uint32) != want.view(np.uint32))
                assert bad.size == 0, (gamma, tier, window, bad[:8], got[bad[:4]], want[bad[:4]])
                for k in COUNTERS:
                    assert st[k] == det["stats"][k], (gamma, tier, window, k)
                pushed = max(pushed, st["push_rounds"])
    assert pushed > n  # sources go past their first round
    g.free()
