"""The FP64 form's tau kernels against the oracle (same operations, same order: equal, no tolerance):
edge counts that choose 8, 16 and 32 edges per warp for the bound, odd edge counts and rows of one
and many forward slots (pairs of edges with one u and with two), eigen row lengths that keep 16-byte
pieces aligned and that do not, and a second run over counters that the first one left."""
from __future__ import annotations

import numpy as np
import pytest

from test_tau_f32_gpu import _csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("omega,uploaded", [(2, 2), (3, 5), (33, 33), (34, 40)])
@pytest.mark.parametrize("n,extra", [(5, 0), (301, 900), (3001, 50000), (4001, 95000)])
def test_taus_and_scores_equal_the_oracle(cuda_device, oracle_lib, omega, uploaded, n, extra):
    from tgtp_b200.aesc import AESC, AESCConfig, AESCGraph, PRECISION_FP64, VEC_F64

    if uploaded > n:
        uploaded = omega = n
    idx, adj = _csr(n, extra, n + omega)
    rng = np.random.default_rng(omega)
    values = np.concatenate([[1.0], np.linspace(0.97, 0.4, uploaded - 1)])
    vec = rng.normal(size=(n, uploaded)) / np.sqrt(n)
    g = AESCGraph.from_csr(idx, adj, values, vec.reshape(-1), VEC_F64)
    sub = np.ascontiguousarray(vec[:, :omega]).reshape(-1)
    for eps in (0.3, 0.3, 0.05):
        a = AESC(g, AESCConfig(eps, omega=omega, precision=PRECISION_FP64))
        got = a.tgtp()
        want, det = oracle_lib.tgtp(idx, adj, values[:omega], sub, eps, fp64=True, details=True)
        assert np.array_equal(a.taus(), det["taus"]), eps
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), eps
        assert a.stats()["tau_iterations"] == det["stats"]["tau_iterations"], eps
        assert a.stats()["push_vertices"] == det["stats"]["push_vertices"], eps
    g.free()
