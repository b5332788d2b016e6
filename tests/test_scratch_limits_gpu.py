"""Calls whose larger working copy does not fit on the device take the smaller one: the walk counters
the plain walk copy and fewer generator states, the mixed form's one-source block push fewer
residual columns at a time.  Same results."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walk", ["saba", "mt", "mt_simd"])
def test_walks_without_room_for_the_packed_copy(cuda_device, oracle_lib, monkeypatch, walk):
    from tgtp_b200 import synth
    from tgtp_b200.aesc import AESCGraph, mt_walk_count, saba_count

    idx, adj = synth.rmat(15, 32, 0.57, 0.19, 0.19, 5).csr()
    m = len(adj)
    depth, walks = 4, 16
    g = AESCGraph.from_csr(idx, adj)
    monkeypatch.setenv("TGTP_ALLOC_LIMIT", str(6 * m))  # 8 bytes a slot packed, 4 plain
    if walk == "saba":
        got = [saba_count(g, depth, walks)[0] for _ in range(2)]
        want = oracle_lib.saba(idx, adj, depth, walks)
    else:
        got = [mt_walk_count(g, depth, walks, simd=walk == "mt_simd")[0] for _ in range(2)]
        want = oracle_lib.mt_walks(idx, adj, depth, walks, simd=walk == "mt_simd")
    g.free()
    for c in got:
        assert np.array_equal(c.astype(np.uint64), want.astype(np.uint64))


def test_block_push_in_several_waves(cuda_device, monkeypatch):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_MIXED, VEC_F32

    n = 20005
    rng = np.random.default_rng(7)
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, 40, n), rng.integers(0, n, 2 * n)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, n), rng.integers(0, n, 2 * n)])
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    values = np.concatenate([[1.0], np.linspace(0.8, 0.5, 15)])
    vec = rng.normal(size=n * 16).astype(np.float32)
    monkeypatch.setenv("TGTP_MIXED_BLOCK", "1")
    got = []
    for limit in (None, 900_000_000):  # all columns take 1.6 GB, two thirds of them more than the limit
        if limit:
            monkeypatch.setenv("TGTP_ALLOC_LIMIT", str(limit))
        g = AESCGraph.from_csr(idx, dst[order].astype(np.uint32), values, vec, VEC_F32)
        a = AESC(g, AESCConfig(0.05, omega=16, gamma=10, precision=PRECISION_MIXED))
        s, again = a.tgtp(), a.tgtp()
        st = a.stats()
        assert np.array_equal(s.view(np.uint32), again.view(np.uint32))
        got.append((s, [st[k] for k in ("push_rounds", "push_vertices", "push_traversals", "walk_edges", "walk_count",
                                        "walk_hops")]))
        g.free()
    assert np.array_equal(got[0][0].view(np.uint32), got[1][0].view(np.uint32)) and got[0][1] == got[1][1]
