"""The FP32 form's tau kernel against the oracle (the same sums in the same order: equal, no
tolerance), where its shape can go wrong: eigen indices around a 32-index step (omega - 1 terms'
ends), fewer pairs used than uploaded, edge counts that are no multiple of 16, sweeps that a whole
warp or few of its edges want, equal rows (a zero dividend), an eigenvalue of 1 beside lambda_0."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, extra, seed):
    rng = np.random.default_rng(seed)
    ring = np.arange(n)
    u = np.concatenate([ring, rng.integers(0, n, extra)])
    v = np.concatenate([(ring + 1) % n, rng.integers(0, n, extra)])
    key = np.unique(np.minimum(u, v).astype(np.int64) * n + np.maximum(u, v))
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    idx = np.zeros(n + 1, np.uint32)
    idx[1:] = np.cumsum(np.bincount(src, minlength=n))
    return idx, dst[order].astype(np.uint32)


PAIRS = [(2, 2), (3, 3), (31, 31), (32, 32), (33, 33), (34, 40), (64, 66), (65, 65), (100, 128)]
GRAPHS = [(5, 0), (37, 60), (301, 900)]


@pytest.mark.parametrize("omega,uploaded,n,extra", [p + g for p in PAIRS for g in GRAPHS if p[1] <= g[0]])
def test_taus_and_scores_equal_the_oracle(cuda_device, oracle_lib, omega, uploaded, n, extra):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, VEC_F32

    idx, adj = _csr(n, extra, n + omega)
    rng = np.random.default_rng(omega)
    values = np.concatenate([[1.0], np.linspace(0.97, 0.4, uploaded - 1)])
    if omega > 4:
        values[2] = 1.0  # no reciprocal of 1 - lambda: the dividends are divided by zero
    vec = (rng.normal(size=(n, uploaded)) / np.sqrt(n)).astype(np.float32)
    vec[::3] = vec[0]  # equal rows: their differences are zero
    if omega > 4:
        vec[:, 2] = rng.normal(size=n).astype(np.float32) if n == 37 else 0.25
    g = AESCGraph.from_csr(idx, adj, values, vec.reshape(-1), VEC_F32)
    sub = np.ascontiguousarray(vec[:, :omega]).reshape(-1)
    for eps in (0.3, 0.05, 0.01):
        a = AESC(g, AESCConfig(eps, omega=omega))
        got = a.tgtp()
        want, det = oracle_lib.tgtp(idx, adj, values[:omega], sub, eps, details=True)
        assert np.array_equal(a.taus(), det["taus"]), (omega, eps)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (omega, eps)
        assert a.stats()["tau_iterations"] == det["stats"]["tau_iterations"], (omega, eps)
    g.free()
