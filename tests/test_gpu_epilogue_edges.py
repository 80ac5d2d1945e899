"""Edges of the update epilogues and of the Grams they form: every rank bucket
(full and one short of full), lengths around whole tiles, and the length
where a launch goes from a block a tile to a warp a tile (296 tiles of 16 rows
/ 32 columns on 148 multiprocessors), against the oracle.

Tolerance: max|d| / max|ref| <= 1e-10 on the factors, the bound of the FP64
path; the HALS family from a start near V's own programs, where it is well
conditioned."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_max

import nmf_rs

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _inputs(n, p, r, seed):
    gen = np.random.default_rng(seed)
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.01
    H = gen.gamma(0.6, 1.0, (r, p)) + 0.01
    V = W @ H * gen.uniform(0.7, 1.3, (n, p))
    V[gen.random((n, p)) < 0.2] = 0.0
    return V, W * gen.uniform(0.8, 1.2, W.shape), H * gen.uniform(0.8, 1.2, H.shape)


def _check(oracle, method, n, p, r, iters=4, **kw):
    V, W0, H0 = _inputs(n, p, r, 1000 * r + n + p)
    ref = oracle.nmf_method(method, V, W0, H0, iters, **kw)
    got = nmf_rs.nmf(V, r, method, W0=W0, H0=H0, max_iter=iters, **kw)
    assert rel_max(got.W, ref["W"]) <= TOL, rel_max(got.W, ref["W"])
    assert rel_max(got.H, ref["H"]) <= TOL, rel_max(got.H, ref["H"])


@pytest.mark.parametrize("method", ["lee", "brunet", "hals", "offset"])
@pytest.mark.parametrize("r", [1, 2, 3, 6, 8, 9, 12, 13, 16, 17, 20, 24, 25, 28, 31, 32])
def test_rank_buckets(oracle, method, r):
    _check(oracle, method, 129, 257, r)


@pytest.mark.parametrize("method", ["lee", "brunet", "hals", "dnmf"])
@pytest.mark.parametrize("n,p", [(15, 31), (16, 32), (17, 33), (33, 1), (4736, 40), (4737, 40),
                                 (40, 9472), (40, 9473), (4753, 9505)])
@pytest.mark.parametrize("r", [5, 32])
def test_tile_edges(oracle, method, n, p, r):
    _check(oracle, method, n, p, min(r, n, max(p, 2)), iters=3)
