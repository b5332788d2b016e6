"""Runs that the device time budget cuts short, at budgets from before the first source to after the
last: each either reports the timeout or gives the complete scores, and the next run on the handle
gives the complete scores, bit for bit (a source that was cut short leaves its residuals in the
block's vector, which in HBM outlives the run)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph():
    n = 6007  # hubs and a sparse rest
    rng = np.random.default_rng(17)
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, 30, n), rng.integers(0, n, n)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, n), rng.integers(0, n, n)])
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


@pytest.mark.parametrize("tier", ["smem", "global"])
@pytest.mark.parametrize("form", ["fp32", "fp64", "mixed"])
def test_a_run_out_of_time_reports_it_and_leaves_the_handle_sound(cuda_device, monkeypatch, form, tier):
    from tgtp_b200._lib import TgtpError
    from tgtp_b200.aesc import (AESC, AESCConfig, AESCGraph, PRECISION_FP32, PRECISION_FP64, PRECISION_MIXED,
                                VEC_F32, VEC_F64)

    idx, adj = _graph()
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.8, 0.5, 15)])
    vec = np.random.default_rng(5).normal(size=n * 16) / np.sqrt(n)
    vec = vec if form == "fp64" else vec.astype(np.float32)
    g = AESCGraph.from_csr(idx, adj, values, vec, VEC_F64 if form == "fp64" else VEC_F32)
    precision = {"fp32": PRECISION_FP32, "fp64": PRECISION_FP64, "mixed": PRECISION_MIXED}[form]
    a = AESC(g, AESCConfig(0.2, omega=16, gamma=10, precision=precision))
    monkeypatch.setenv("TGTP_PVEC_TIER", tier)
    monkeypatch.setenv("TGTP_MIXED_BLOCK", "0")
    want = a.tgtp()
    cut = 0
    for budget in ("1e-9", "2e-6", "5e-6", "1e-5", "2e-5", "4e-5", "8e-5", "1.6e-4", "3.2e-4", "6.4e-4", "1.3e-3"):
        monkeypatch.setenv("TGTP_KERNEL_DEADLINE_S", budget)
        for _ in range(3):
            try:
                assert np.array_equal(a.tgtp().view(np.uint32), want.view(np.uint32)), budget
            except TgtpError as e:
                assert "time budget" in str(e)
                cut += 1
        monkeypatch.delenv("TGTP_KERNEL_DEADLINE_S")
        assert np.array_equal(a.tgtp().view(np.uint32), want.view(np.uint32)), budget
    assert cut >= 9  # the shortest budgets end inside the run
    g.free()
