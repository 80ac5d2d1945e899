"""Edges of the kernels for ranks above 32: ranks around whole 8-column Gram
tiles (the column of ones included), 4-entry update groups and the 64 tiles of
a Gram block; lengths around the 32-line updates, the 32-row Gram chunks and
the 128 x 64 tiles of W H; against the oracle.

Tolerance: max|d| / max|ref| <= 1e-10 on the factors, the FP64 path's bound;
the HALS family from a start near V's own programs."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_max

import nmf_rs

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _run(oracle, method, n, p, r, iters=3, **kw):
    gen = np.random.default_rng(n + 3 * p + 11 * r)
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.01
    H = gen.gamma(0.6, 1.0, (r, p)) + 0.01
    V = W @ H * gen.uniform(0.7, 1.3, (n, p))
    V[gen.random((n, p)) < 0.2] = 0.0
    W0, H0 = W * gen.uniform(0.8, 1.2, W.shape), H * gen.uniform(0.8, 1.2, H.shape)
    ref = oracle.nmf_method(method, V, W0, H0, iters, **kw)
    got = nmf_rs.nmf(V, r, method, W0=W0, H0=H0, max_iter=iters, **kw)
    assert rel_max(got.W, ref["W"]) <= TOL, rel_max(got.W, ref["W"])
    assert rel_max(got.H, ref["H"]) <= TOL, rel_max(got.H, ref["H"])
    return got, ref


@pytest.mark.parametrize("method,r", [
    (m, r) for m in ("lee", "brunet", "hals", "dnmf")
    for r in (33, 34, 35, 39, 40, 47, 64, 87, 88, 129, 256)
    if (m, r) != ("hals", 256)])  # at 300 rows the oracle itself moves by 2e-2 a one-ulp change
def test_ranks(oracle, method, r):
    _run(oracle, method, 300, 330, r)


@pytest.mark.parametrize("method", ["lee", "brunet", "hals"])
@pytest.mark.parametrize("n,p", [(63, 64), (127, 65), (128, 129), (129, 63), (257, 97), (97, 1025)])
def test_lengths(oracle, method, n, p):
    _run(oracle, method, n, p, 37)


@pytest.mark.parametrize("method", ["lee", "brunet"])
@pytest.mark.parametrize("n,p", [(127, 65), (129, 63)])
def test_deviances(oracle, method, n, p):
    got, ref = _run(oracle, method, n, p, 41, stop="stationary", stationary_th=0.0)
    assert got.n_iter == ref["n_iter"]
    np.testing.assert_allclose(got.deviances, ref["deviances"], rtol=1e-11)


@pytest.mark.parametrize("r", [34, 41])
@pytest.mark.parametrize("k", [0, 9])
@pytest.mark.parametrize("scale,size", [(2.0 ** -535, np.float64(1e150)), (2.0 ** -560, np.inf)])
def test_vanishing_component(oracle, r, k, scale, size):
    """eps = 0 and a column of W whose squares add up to a subnormal (64 x
    2^-1070, exact) or to 0: H's row is the quotient by that, huge or infinite,
    not eps."""
    gen = np.random.default_rng(7 * r + k)
    n, p = 64, 70
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.01
    H = 1e-3 * gen.gamma(0.6, 1.0, (r, p))
    W[:, k] = scale
    V = 1e3 + gen.random((n, p))  # far above W H: the row's own sum stays positive
    if k:  # ... and the components before it are empty
        W[:, :k] = 0.0
        H[:k] = 0.0
    ref = oracle.nmf_method("hals", V, W, H, 1, eps=0.0)
    got = nmf_rs.nmf(V, r, "hals", W0=W, H0=H, max_iter=1, eps=0.0)
    assert ref["H"][k].min() > size if size < np.inf else np.all(ref["H"][k] == np.inf)
    for a, b in ((got.W, ref["W"]), (got.H, ref["H"])):
        np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    if size == np.inf:
        assert np.all(got.H[k] == np.inf)
    else:
        # the module's bound, on the row itself
        assert rel_max(got.H[k], ref["H"][k]) <= TOL
