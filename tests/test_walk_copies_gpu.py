"""The walk copies of saba_count and mt_walk_count (packed: 8 bytes per slot and a table of degree
classes; plain: for graphs with more classes than the table holds) against the CPU oracle: every
counter equal, so no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, u, v):
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


def _graph(name):
    from tgtp_b200 import synth

    if name == "one_class":  # a ring: every degree 2
        r = np.arange(33)
        return _csr(33, r, (r + 1) % 33)
    if name == "isolated":  # ids without an edge among the others
        return _csr(40, np.array([3, 3, 3, 17, 17, 38]), np.array([17, 20, 38, 20, 21, 21]))
    if name == "repeats":  # repeated edges and a self-loop
        return _csr(5, np.array([0, 0, 0, 1, 2, 2, 3]), np.array([1, 1, 2, 2, 3, 2, 4]))
    if name == "classes":  # 4,199 distinct degrees: beyond the class table
        n = 4200
        u = np.repeat(np.arange(n), n)
        v = np.tile(np.arange(n), n)
        keep = (u < v) & (u + v >= n - 1)
        return _csr(n, u[keep], v[keep])
    return synth.rmat(12, 8, 0.57, 0.19, 0.19, 5).csr()


@pytest.mark.parametrize("name", ["one_class", "isolated", "repeats", "classes", "rmat12"])
@pytest.mark.parametrize("depth,walks", [(1, 8), (5, 24), (11, 136)])
def test_saba_over_each_kind_of_copy(cuda_device, oracle_lib, name, depth, walks):
    from tgtp_b200.aesc import AESCGraph, saba_count

    idx, adj = _graph(name)
    g = AESCGraph.from_csr(idx, adj)
    counts, visits, checksum, _ = saba_count(g, depth, walks)
    again = saba_count(g, depth, walks)
    g.free()
    want = oracle_lib.saba(idx, adj, depth, walks)
    assert np.array_equal(counts.astype(np.uint64), want) and np.array_equal(counts, again[0])
    assert visits == int(want.sum())
    assert checksum == int((want * np.arange(1, len(want) + 1, dtype=np.uint64)).sum())


@pytest.mark.parametrize("simd", [False, True])
@pytest.mark.parametrize("name,depth,walks", [
    ("one_class", 5, 264), ("isolated", 2, 1000), ("repeats", 7, 16), ("classes", 3, 8),
    # walks side by side: all 128, 124, 33, 32, 9 (a walk takes 78 draws), one; tails of each
    ("rmat12", 2, 264), ("rmat12", 5, 136), ("rmat12", 19, 72), ("rmat12", 20, 40), ("rmat12", 78, 16),
    ("rmat12", 624, 8)])
def test_mt_walks_over_each_kind_of_copy(cuda_device, oracle_lib, simd, name, depth, walks):
    from tgtp_b200.aesc import AESCGraph, mt_walk_count

    idx, adj = _graph(name)
    g = AESCGraph.from_csr(idx, adj)
    counts, visits, _ = mt_walk_count(g, depth, walks, simd=simd)
    g.free()
    want = oracle_lib.mt_walks(idx, adj, depth, walks, simd=simd)
    assert np.array_equal(counts.astype(np.uint64), want)
    assert visits == int(want.sum())
