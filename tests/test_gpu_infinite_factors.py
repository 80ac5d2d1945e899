"""Infinite factor entries.  A term past V's edge has one operand of 0 and an
entry of a factor as the other, and 0 * inf is NaN: sizes off the tiles give
what whole tiles give, the oracle's value."""
from __future__ import annotations

import numpy as np
import pytest

import nmf_rs
from nmf_rs import _native

pytestmark = pytest.mark.gpu


def _inputs(n, p, r):
    """V near W H, all factor entries positive (0 * inf is NaN in the oracle too)."""
    gen = np.random.default_rng(n + 5 * p + 11 * r)
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.01
    H = gen.gamma(0.6, 1.0, (r, p)) + 0.01
    return W @ H * gen.uniform(0.7, 1.3, (n, p)), W, H


def _infinite(side, V, W, H):
    """The last row's W, or the last column's H, infinite; V is 0 there, where
    KL's term is W H itself."""
    if side == "w":
        W[-1, 1] = np.inf
        V[-1] = 0.0
    else:
        H[1, -1] = np.inf
        V[:, -1] = 0.0


# 16-row units; 256-column tiles up to rank 24, 128 above
SIZES = [(16, 256), (17, 256), (16, 257), (15, 127), (33, 129), (40, 300)]


@pytest.mark.parametrize("side", ["w", "h"])
@pytest.mark.parametrize("r", [2, 10, 24, 28])
@pytest.mark.parametrize("n,p", SIZES)
def test_objective_is_infinite(oracle, n, p, r, side):
    V, W, H = _inputs(n, p, r)
    _infinite(side, V, W, H)
    assert oracle.kl_divergence(V, W, H) == np.inf == oracle.euclidean_distance(V, W, H)
    assert _native.divergence(V, W, H) == np.inf
    assert _native.distance(V, W, H) == np.inf


@pytest.mark.parametrize("method", ["lee", "hals", "offset"])
@pytest.mark.parametrize("n,p", [(17, 33), (16, 257), (33, 256)])
def test_stationary_run_goes_on(oracle, method, n, p):
    """An infinite objective does not end a run (a NaN does)."""
    V, W, H = _inputs(n, p, 3)
    H[1, 5] = np.inf
    kw = dict(stop="stationary", stationary_th=0.0)
    ref = oracle.nmf_method(method, V, W, H, 3, **kw)
    got = nmf_rs.nmf(V, 3, method, W0=W, H0=H, max_iter=3, **kw)
    assert got.n_iter == ref["n_iter"] and ref["n_iter"] > 0
    np.testing.assert_allclose(got.deviances, ref["deviances"], rtol=1e-9)


# ranks above 32: 128 x 64 tiles
@pytest.mark.parametrize("method", ["lee", "brunet", "hals"])
@pytest.mark.parametrize("side", ["w", "h"])
@pytest.mark.parametrize("n,p", [(128, 64), (129, 64), (128, 65), (100, 110), (130, 261)])
def test_wide_objective_is_infinite(oracle, method, side, n, p):
    V, W, H = _inputs(n, p, 34)
    _infinite(side, V, W, H)
    kw = dict(stop="stationary", stationary_th=0.0)
    ref = oracle.nmf_method(method, V, W, H, 1, **kw)
    got = nmf_rs.nmf(V, 34, method, W0=W, H0=H, max_iter=1, **kw)
    assert ref["deviances"][0] == np.inf == got.deviances[0]
    assert got.n_iter == ref["n_iter"] == 1
