"""The FP32 and FP64 forms' edge bound where gamma (above 64) exceeds the number of positive
residuals of the frontier but not its size: the gamma-th largest residual is then 0.  Against the
oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _windmill(k):
    """k triangles that share vertex 0.  The sequential push drains a triangle's second leaf after
    its first one has reached it, so about half of the frontier holds residual 0."""
    n = 2 * k + 1
    a = np.arange(1, n, 2)
    hub = np.zeros(k, np.int64)
    u, v = np.concatenate([hub, hub, a]), np.concatenate([a, a + 1, a + 1])
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


@pytest.mark.parametrize("fp64", [False, True], ids=["fp32", "fp64"])
def test_rank_beyond_the_positive_residuals(cuda_device, oracle_lib, monkeypatch, fp64):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_FP32, PRECISION_FP64, VEC_F32, VEC_F64

    idx, adj = _windmill(200)  # frontiers of 401 vertices, 201 or 400 of them positive
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.97, 0.67, 15)])
    vec = np.random.default_rng(5).normal(size=(n, 16)) * 2.0
    vec[:21] = 0.0  # the hub and ten triangles keep their long walks, the others lose most of theirs
    vec = vec.reshape(-1) if fp64 else vec.reshape(-1).astype(np.float32)
    g = AESCGraph.from_csr(idx, adj, values, vec, VEC_F64 if fp64 else VEC_F32)
    for gamma in (65, 201, 202, 300, 400):
        want, det = oracle_lib.tgtp(idx, adj, values, vec, 0.3, gamma=gamma, fp64=fp64, details=True)
        assert det["stats"]["walk_edges"] > 100  # slots walk, so the bound is used
        for tier in ("smem", "global"):
            monkeypatch.setenv("TGTP_PVEC_TIER", tier)
            a = AESC(g, AESCConfig(0.3, omega=16, gamma=gamma, precision=PRECISION_FP64 if fp64 else PRECISION_FP32))
            got = a.tgtp()
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (gamma, tier)
            st = a.stats()
            for k in ("push_rounds", "walk_edges", "walk_count", "walk_hops"):
                assert st[k] == det["stats"][k], (gamma, tier, k)
    g.free()
