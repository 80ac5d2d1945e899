"""Infinite factor entries.  A term past V's edge has one operand of 0 and an
entry of a factor as the other, and 0 * inf is NaN: sizes off the tiles give
what whole tiles give, the oracle's value."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

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


@pytest.mark.parametrize("r", [20, 34])
@pytest.mark.parametrize("v", [np.inf, -np.inf])
def test_infinite_entry(oracle, r, v):
    """The ratio of an infinite entry of V keeps its sign (py_nmf_run, like the
    reference's, takes a V of any sign; nmf() itself refuses a negative one)."""
    V, W, H = _inputs(50, 70, r)
    V[3, 5] = v
    ref = oracle.nmf_method("brunet", V, W, H, 1)
    got = _native.py_nmf_run("brunet", V, W, H, 1)
    assert np.all(ref["H"][:, 5] == v)
    np.testing.assert_array_equal(np.isfinite(got["H"]), np.isfinite(ref["H"]))
    np.testing.assert_array_equal(got["H"][:, 5], ref["H"][:, 5])


def _stored_brunet(M, W, H):
    """One brunet iteration over the stored entries of M alone."""
    c = M.tocoo()
    i, j, v = c.row, c.col, c.data

    def quotient(W, H):
        wh = (W[i] * H[:, j].T).sum(1)
        return np.where(wh != 0.0, v / np.where(wh != 0.0, wh, 1.0), 0.0)

    with np.errstate(all="ignore"):
        num = np.zeros((H.shape[1], H.shape[0]))
        np.add.at(num, j, quotient(W, H)[:, None] * W[i])
        H = H * num.T / W.sum(0)[:, None]
        num = np.zeros(W.shape)
        np.add.at(num, i, quotient(W, H)[:, None] * H[:, j].T)
        return W * num / H.sum(1)[None, :], H


# Lines that gather (the lower ranks, the sparser ones) and lines with enough
# entries for the blocked passes.
@pytest.mark.parametrize("side", ["w", "h"])
@pytest.mark.parametrize("n,p,r,density", [(150, 170, 2, 0.5), (301, 500, 4, 0.6),
                                           (300, 500, 6, 0.6), (1100, 2200, 20, 0.2),
                                           (900, 1000, 32, 0.2), (700, 1500, 20, 0.01)])
def test_sparse_lines_keep_infinity(n, p, r, density, side):
    """V / (W H) is 0 at a stored entry whose W H is infinite, whatever the
    number of entries of its line."""
    V, W, H = _inputs(n, p, r)
    V[np.random.default_rng(2).random(V.shape) >= density] = 0.0
    if side == "w":
        W[7, 1] = np.inf
    else:
        H[1, 9] = np.inf
    M = sp.csr_matrix(V)
    want_W, want_H = _stored_brunet(M, W, H)
    got = nmf_rs.nmf(M, r, "brunet", W0=W, H0=H, max_iter=1)
    for g, w in ((got.W, want_W), (got.H, want_H)):
        np.testing.assert_array_equal(np.isnan(g), np.isnan(w))
        # the FP64 path's bound, 1e-10 of the largest
        ok = np.isfinite(w)
        assert np.all(np.abs(g[ok] - w[ok]) <= 1e-10 * np.abs(w[ok]).max(initial=0.0))
