"""Edges of the FP64 objective pass: lengths around its 16-row units and
256-column tiles (128 above rank 24), every kind of element (v = 0, W H = 0,
ratios from 1e-300 to 1e300 and near 1), against the oracle.

Tolerance: relative 1e-12, the objective's bound in the FP64 path, plus the
rounding floor of the sums, 10 eps sum(V)."""
from __future__ import annotations

import numpy as np
import pytest

import nmf_rs
from nmf_rs import _native

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _near(a, b, floor):
    if not np.isfinite(b):  # infinite quotients: the oracle's sum has no finite value either
        assert a == b or (np.isnan(a) and np.isnan(b)), (a, b)
        return
    assert abs(a - b) <= 1e-12 * abs(b) + 10 * EPS * floor, (a, b)


@pytest.mark.parametrize("r", [1, 4, 10, 20, 25, 32])
@pytest.mark.parametrize("n,p", [(1, 1), (15, 255), (16, 256), (17, 257), (33, 128), (40, 129),
                                 (700, 90), (64, 3000)])
def test_objectives_match_the_oracle(oracle, n, p, r):
    gen = np.random.default_rng(n + 7 * p + r)
    W = gen.gamma(0.5, 1.0, (n, r))
    H = gen.gamma(0.5, 1.0, (r, p))
    V = (W @ H) * np.exp(gen.normal(0.0, 1.0, (n, p)))
    V[gen.random((n, p)) < 0.3] = 0.0
    W[0] = 0.0          # W H = 0 under positive and zero entries
    if n > 2:
        V[1] = (W @ H)[1]  # ratios of 1
    _near(_native.divergence(V, W, H), oracle.kl_divergence(V, W, H), V.sum() + (W @ H).sum())
    _near(_native.distance(V, W, H), oracle.euclidean_distance(V, W, H), (V * V).sum())


def test_extreme_ratios(oracle):
    """Quotients at both ends of the range, subnormal W H among them."""
    e = np.array([-305.0, -290.0, -150.0, -3.0, -1e-9, 0.0, 1e-12, 0.3, 0.35, 2.0, 100.0, 290.0])
    V = np.repeat((10.0 ** np.clip(e, -200, 200))[None, :], 3, axis=0)
    W = np.array([[1.0], [1e-100], [3.0]])
    H = (10.0 ** np.clip(-e, -200, 200))[None, :]
    H[0, 2] = 5e-324
    _near(_native.divergence(V, W, H), oracle.kl_divergence(V, W, H),
          np.abs(V).sum() + np.abs(W @ H).sum())
    for j in range(e.size):  # and by itself, so that no column hides another
        v, h = np.ascontiguousarray(V[:, j:j + 1]), np.ascontiguousarray(H[:, j:j + 1])
        _near(_native.divergence(v, W, h), oracle.kl_divergence(v, W, h), v.sum() + (W @ h).sum())


@pytest.mark.parametrize("method", ["offset", "nsNMF"])
def test_deviances_of_offset_and_nsnmf(oracle, method):
    """The row offsets (no term past V's last column) and W S in the pass."""
    gen = np.random.default_rng(3)
    V = gen.gamma(1.0, 1.0, (45, 270)) + 0.01
    W0, H0 = nmf_rs.random_init(V, 5, seed=1)
    kw = dict(stop="stationary", stationary_th=0.0)
    got = nmf_rs.nmf(V, 5, method, W0=W0, H0=H0, max_iter=6, **kw)
    ref = oracle.nmf_method(method, V, W0, H0, 6, **kw)
    assert got.n_iter == ref["n_iter"]
    np.testing.assert_allclose(got.deviances, ref["deviances"], rtol=1e-11)
