"""Captured runs that use the handle's own scratch (a batch with TGTP_BATCH_PERSISTENT=0, or a mixed run
that takes a block push) between plain runs of another form on the same handle.  Both sides keep their
residual vectors zeroed in HBM from one run to the next, in one scratch carved in two ways: each run
has to see the other's.  Scores bit for bit those of a handle of its own."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph():
    n = 3001
    rng = np.random.default_rng(23)
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, 20, n), rng.integers(0, n, n)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, n), rng.integers(0, n, n)])
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


@pytest.mark.parametrize("captured,plain,block", [("fp32", "fp64", "0"), ("mixed", "fp64", "0"), ("fp64", "mixed", "0"),
                                                  ("mixed", "fp64", "1")])
def test_replays_and_plain_runs_do_not_trust_each_others_scratch(cuda_device, monkeypatch, captured, plain, block):
    import torch

    from tgtp_b200.aesc import (AESC, AESCConfig, AESCGraph, Batch, PRECISION_FP32, PRECISION_FP64, PRECISION_MIXED,
                                VEC_F32, VEC_F64)

    monkeypatch.setenv("TGTP_PVEC_TIER", "global")
    monkeypatch.setenv("TGTP_MIXED_BLOCK", block)
    if block == "0":
        monkeypatch.setenv("TGTP_BATCH_PERSISTENT", "0")
    form = {"fp32": PRECISION_FP32, "fp64": PRECISION_FP64, "mixed": PRECISION_MIXED}
    idx, adj = _graph()
    n = len(idx) - 1
    values = np.concatenate([[1.0], np.linspace(0.8, 0.5, 15)])
    vec = np.random.default_rng(5).normal(size=n * 16).astype(np.float32) / np.float32(np.sqrt(n))

    def handle():
        g = AESCGraph.from_csr(idx, adj)
        g.upload_eigens(values, vec, VEC_F32)
        g.upload_eigens(values, vec.astype(np.float64), VEC_F64)
        return g

    want = {}
    for f in (captured, plain):
        g = handle()
        want[f] = AESC(g, AESCConfig(0.2, omega=16, gamma=10, precision=form[f])).tgtp().view(np.uint32)
        g.free()
    g = handle()
    run = AESC(g, AESCConfig(0.2, omega=16, gamma=10, precision=form[plain]))
    for f in ("mixed", "fp64", "fp32"):  # every buffer at its largest before the batch pins them
        AESC(g, AESCConfig(0.2, omega=16, gamma=10, precision=form[f])).tgtp()
    assert np.array_equal(run.tgtp().view(np.uint32), want[plain])
    out = torch.empty(g.m, dtype=torch.float32, device="cuda")
    batch = Batch([(AESC(g, AESCConfig(0.2, omega=16, gamma=10, precision=form[captured])), out.data_ptr())])
    for _ in range(2):
        assert np.array_equal(run.tgtp().view(np.uint32), want[plain])
        for _ in range(2):
            out.zero_()
            torch.cuda.synchronize()
            batch.run()
            batch.wait()
            assert np.array_equal(out.cpu().numpy().view(np.uint32), want[captured])
    batch.free()
    assert np.array_equal(run.tgtp().view(np.uint32), want[plain])
    g.free()
