"""Calls whose larger working copy does not fit on the device take the smaller one: the walk counters
the plain walk copy and fewer generator states.  Same results."""
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
