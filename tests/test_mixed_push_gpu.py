"""The mixed form's pushes against one another (each sums residuals exactly, so scores and work
counters are equal bit for bit, no tolerance): one source per block in shared memory, 32 sources per
CTA as a pull product, and the per-source kernel, on graphs at the sizes where the shared-memory
push changes: rows of 255 .. 257 entries (light and heavy vertices), frontiers of more than 512
heavy vertices, 256 / 512 / 1,024 threads per block, vertex counts that are no multiple of 32."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTERS = ("push_rounds", "push_vertices", "push_traversals", "walk_edges", "walk_count", "walk_hops")


def _csr(n, u, v):
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    keep = u != v
    u, v = u[keep], v[keep]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


def _graph(name):
    rng = np.random.default_rng(7)
    if name == "rows255-257":  # three hubs of exactly 255, 256 and 257 neighbours
        n = 801
        ring = np.arange(n)
        u, v = [ring], [(ring + 1) % n]
        for hub, deg in ((10, 255), (20, 256), (30, 257)):
            others = np.setdiff1d(np.arange(40, n), [hub - 1, hub + 1])[: deg - 2]
            u.append(np.full(len(others), hub))
            v.append(others)
        return _csr(n, np.concatenate(u), np.concatenate(v))
    if name == "heavy":  # 700 vertices of about 300 neighbours
        n = 1031
        u = np.repeat(np.arange(700), 215)
        return _csr(n, u, rng.integers(0, n, u.size))
    n = {"mid": 7003, "wide": 20005}[name]  # hubs and a sparse rest
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, 40, n), rng.integers(0, n, 2 * n)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, n), rng.integers(0, n, 2 * n)])
    return _csr(n, u, v)


def _run(g, eps, gamma):
    from tgtp_b200.aesc import AESC, AESCConfig, PRECISION_MIXED

    a = AESC(g, AESCConfig(eps, omega=16, gamma=gamma, precision=PRECISION_MIXED))
    s = a.tgtp()
    st = a.stats()
    return s, {k: st[k] for k in COUNTERS}


@pytest.mark.parametrize("name", ["rows255-257", "heavy", "mid", "wide"])
@pytest.mark.parametrize("gamma", [1, 10, 40])
def test_every_push_gives_the_same_bits(cuda_device, monkeypatch, name, gamma):
    from tgtp_b200.aesc import AESCGraph, VEC_F32

    idx, adj = _graph(name)
    rng = np.random.default_rng(3)
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.8, 0.5, 15)])
    vectors = rng.normal(size=n * 16).astype(np.float32)
    g = AESCGraph.from_csr(idx, adj, values, vectors, VEC_F32)
    for eps in (0.05, 0.01, 0.001):
        got = {}
        for push, env in (("source", {"TGTP_MIXED_BLOCK": "0"}), ("block", {"TGTP_MIXED_BLOCK": "1"}),
                          ("source_hbm", {"TGTP_MIXED_BLOCK": "0", "TGTP_PVEC_TIER": "global"}),
                          ("block32", {"TGTP_MIXED_BLOCK": "1", "TGTP_BLOCK_CTAS": "148"})):
            for k in ("TGTP_MIXED_BLOCK", "TGTP_BLOCK_CTAS", "TGTP_PVEC_TIER"):
                monkeypatch.delenv(k, raising=False)
            for k, v in env.items():
                monkeypatch.setenv(k, v)
            got[push] = _run(g, eps, gamma)
            again = _run(g, eps, gamma)
            assert np.array_equal(again[0].view(np.uint32), got[push][0].view(np.uint32)), push
        for push in ("source", "source_hbm", "block32"):
            assert np.array_equal(got["block"][0].view(np.uint32), got[push][0].view(np.uint32)), push
            assert got["block"][1] == got[push][1], push
    assert got["block"][1]["push_rounds"] > n  # rows push past their first round
    g.free()
