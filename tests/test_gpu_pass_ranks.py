"""The FP64 passes at ranks on and off their tiles of 8, over several tiles,
boxes and units; and the quotient V / (W H) at the ends of its fast range.

Tolerances: max|d| / max|ref| <= 1e-10 on the factors, the FP64 path's bound;
for one quotient at rank 1, 16 eps: the product, the quotient (an ulp against
half), the two products and the division around it, each below an ulp."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_max

import nmf_rs
from nmf_rs import _native

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("method", ["lee", "brunet", "lsnmf"])
@pytest.mark.parametrize("n,p", [(530, 1030), (1025, 513), (17, 2100)])
@pytest.mark.parametrize("r", [2, 4, 10, 12, 18, 20, 26, 28])
def test_pass_ranks(oracle, method, n, p, r):
    r = min(r, n)
    gen = np.random.default_rng(100 * r + n)
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.01
    H = gen.gamma(0.6, 1.0, (r, p)) + 0.01
    V = W @ H * gen.uniform(0.7, 1.3, (n, p))
    V[gen.random((n, p)) < 0.2] = 0.0
    W0, H0 = W * gen.uniform(0.8, 1.2, W.shape), H * gen.uniform(0.8, 1.2, H.shape)
    if method == "lsnmf":
        S = gen.uniform(0.5, 1.5, V.shape)
        ref = oracle.nmf_lsnmf(V, S, W0, H0, 3)
        got = nmf_rs.nmf(V, r, method, W0=W0, H0=H0, max_iter=3, weight=S)
    else:
        ref = oracle.nmf_method(method, V, W0, H0, 3)
        got = nmf_rs.nmf(V, r, method, W0=W0, H0=H0, max_iter=3)
    assert rel_max(got.W, ref["W"]) <= 1e-10
    assert rel_max(got.H, ref["H"]) <= 1e-10


@pytest.mark.parametrize("side", ["h", "w"])
@pytest.mark.parametrize("v", [0.0, 1.0, 3.7e-5, np.inf, np.nan])
def test_quotient_range(oracle, v, side):
    # W H across the doubles: subnormal, around 2^-1000 and 2^1000, infinite.
    y = np.concatenate([[0.0, 5e-324, 1e-310, 2.0 ** -1000, 2.0 ** 1000, 1.7e308, np.inf],
                        2.0 ** np.arange(-1004.5, -995.5), 2.0 ** np.arange(995.5, 1004.5),
                        10.0 ** np.linspace(-12, 12, 41)])
    m = y.size
    if side == "h":
        args = np.full((1, m), v), np.ones((1, 1)), y[None, :].copy()
        got, want = _native.py_divergence_update_h(*args), oracle.update_h_brunet(*args)
    else:
        args = np.full((m, 1), v), y[:, None].copy(), np.ones((1, 1))
        got, want = _native.py_divergence_update_w(*args), oracle.update_w_brunet(*args)
    got, want = np.asarray(got).ravel(), np.asarray(want).ravel()
    fin = np.isfinite(want)
    np.testing.assert_array_equal(got[~fin], want[~fin])
    assert np.all(np.abs(got[fin] - want[fin]) <= 16 * EPS * np.abs(want[fin])), (got, want)
