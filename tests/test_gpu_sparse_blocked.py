"""The sparse passes that keep blocks of factor rows in shared memory: several
blocks with a remainder, every rank bucket, empty and full lines, lines of few
entries (which take the gathering passes), and unsorted rows; against the dense
oracle, max|d| / max|ref| <= 1e-10, the FP64 path's bound."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from conftest import rel_max

import nmf_rs
from nmf_rs import _native

pytestmark = pytest.mark.gpu
TOL = 1e-10


def _inputs(n, p, r, density, seed):
    gen = np.random.default_rng(seed)
    W = gen.gamma(0.6, 1.0, (n, r)) + 0.05
    H = gen.gamma(0.6, 1.0, (r, p)) + 0.05
    V = W @ H * gen.uniform(0.7, 1.3, (n, p))
    V[gen.random((n, p)) >= density] = 0.0
    return V, W * gen.uniform(0.8, 1.2, W.shape), H * gen.uniform(0.8, 1.2, H.shape)


def _check(oracle, method, V, W0, H0, iters=3):
    ref = oracle.nmf_method(method, V, W0, H0, iters)
    got = nmf_rs.nmf(sp.csr_matrix(V), W0.shape[1], method, W0=W0, H0=H0, max_iter=iters)
    assert rel_max(got.W, ref["W"]) <= TOL, rel_max(got.W, ref["W"])
    assert rel_max(got.H, ref["H"]) <= TOL, rel_max(got.H, ref["H"])


# 204800 / (8 rank) factor rows a block, down to a multiple of 32: 800 at rank
# 32, 1280 at 20, 3200 at 8, 12800 at 2
@pytest.mark.parametrize("method", ["lee", "brunet"])
@pytest.mark.parametrize("n,p,r,density", [
    (801, 1601, 32, 0.1), (1600, 900, 30, 0.1), (930, 1000, 28, 0.2), (1100, 2200, 23, 0.08),
    (1281, 2561, 20, 0.06), (1700, 1650, 16, 0.05), (400, 1900, 14, 0.3), (300, 2200, 12, 0.3),
    (2600, 300, 10, 0.3), (3201, 200, 8, 0.4), (200, 4400, 6, 0.4), (150, 6500, 4, 0.5),
    (60, 12801, 2, 0.5), (500, 500, 1, 0.5)])
def test_blocks_and_ranks(oracle, method, n, p, r, density):
    V, W0, H0 = _inputs(n, p, r, density, n + p + r)
    if method == "brunet":  # brunet divides by W H only where V is stored
        V[:, V.sum(0) == 0] += 0.01
    _check(oracle, method, V, W0, H0)


def test_empty_and_full_lines(oracle):
    V, W0, H0 = _inputs(1300, 1400, 20, 0.1, 5)
    V[::7] = 0.0
    V[3] = 1.5
    V[:, 11] = 0.25
    V[:, 100:140] = 0.0
    _check(oracle, "lee", V, W0, H0)


def test_few_entries(oracle):
    """Rows of 15 entries a block and columns below it: the gathering passes."""
    V, W0, H0 = _inputs(700, 1500, 20, 0.01, 6)
    _check(oracle, "lee", V, W0, H0)


@pytest.mark.parametrize("method", ["lee", "brunet"])
def test_unsorted_rows(method):
    """Rows whose entries are not in column order give the same factors."""
    n, p, r, iters = 1300, 1500, 20, 3
    V, W0, H0 = _inputs(n, p, r, 0.1, 9)
    M = sp.csr_matrix(V)
    want = nmf_rs.nmf(M, r, method, W0=W0, H0=H0, max_iter=iters)
    gen = np.random.default_rng(1)
    idx, dat = M.indices.astype(np.int32), M.data.copy()
    for i in range(n):
        a, b = M.indptr[i], M.indptr[i + 1]
        o = gen.permutation(b - a)
        idx[a:b], dat[a:b] = idx[a:b][o], dat[a:b][o]
    ptr = M.indptr.astype(np.int64)
    o = _native.default_options()
    o.method = _native.parse_method(method)
    o.max_iter = iters
    W, H = np.empty_like(W0), np.empty_like(H0)
    nd, ni = ctypes.c_int64(0), ctypes.c_int64(0)
    _native.check(_native.load().nmfcu_run_csr(
        ctypes.byref(o), n, p, r, dat.size, ptr.ctypes.data_as(_native._i64p),
        idx.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), _native._ptr(dat),
        _native._ptr(W0), _native._ptr(H0), _native._ptr(W), _native._ptr(H), None, 0,
        ctypes.byref(nd), ctypes.byref(ni)))
    assert rel_max(W, want.W) <= TOL and rel_max(H, want.H) <= TOL


# Above 2^22 entries the CSC copy is made by 128 x 2048 tiles, 256 columns of
# one at a time: one row and a few columns past whole tiles; nearly full ones,
# whose sub-tiles hold more entries than their lists; rows of one tile.
@pytest.mark.parametrize("n,p,density", [(2177, 4099, 0.5), (1500, 3300, 0.9), (100, 50001, 0.9),
                                         (40001, 300, 0.4)])
def test_csc_tiles(oracle, n, p, density):
    V, W0, H0 = _inputs(n, p, 3, density, n + p)
    assert np.count_nonzero(V) > 1 << 22
    _check(oracle, "lee", V, W0, H0, iters=2)


@pytest.mark.parametrize("n,p", [(127, 2047), (1, 300), (700, 3)])
def test_csc_sort(oracle, n, p):
    V, W0, H0 = _inputs(n, p, 3, 0.15, n + p)
    V[0, 0] = V[-1, -1] = 1.0
    _check(oracle, "lee", V, W0, H0)


def test_repeated_entries():
    """Two stored entries of one place count as their sum (lee: linear in V)."""
    n, p, r = 300, 500, 4
    V, W0, H0 = _inputs(n, p, r, 0.2, 4)
    M = sp.csr_matrix(V)
    want = nmf_rs.nmf(M, r, "lee", W0=W0, H0=H0, max_iter=3)
    ptr = (2 * M.indptr).astype(np.int64)
    idx = np.repeat(M.indices, 2).astype(np.int32)
    dat = np.repeat(M.data / 2, 2)
    o = _native.default_options()
    o.method = _native.parse_method("lee")
    o.max_iter = 3
    W, H = np.empty_like(W0), np.empty_like(H0)
    nd, ni = ctypes.c_int64(0), ctypes.c_int64(0)
    _native.check(_native.load().nmfcu_run_csr(
        ctypes.byref(o), n, p, r, dat.size, ptr.ctypes.data_as(_native._i64p),
        idx.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), _native._ptr(dat),
        _native._ptr(W0), _native._ptr(H0), _native._ptr(W), _native._ptr(H), None, 0,
        ctypes.byref(nd), ctypes.byref(ni)))
    assert rel_max(W, want.W) <= TOL and rel_max(H, want.H) <= TOL


def _launches(n, p, r, density, method="lee"):
    """Kernels of a run of no iterations over a device CSR."""
    return _launches_of(sp.csr_matrix(_inputs(n, p, r, density, 3)[0]), r, method)


def _launches_of(M, r, method):
    n, p = M.shape
    W0, H0 = np.ones((n, r)), np.ones((r, p))
    dev = [torch.from_numpy(x).cuda() for x in
           (M.indptr.astype(np.int64), M.indices.astype(np.int32), M.data, W0, H0)]
    o = _native.default_options()
    o.method = _native.parse_method(method)
    o.max_iter = 0
    ctx = _native.Context(0)
    nd, ni = ctypes.c_int64(0), ctypes.c_int64(0)
    at = [ctypes.c_void_p(x.data_ptr()) for x in dev]
    before = ctx.launch_count()
    _native.check(_native.load().nmfcu_run_csr_device(
        ctx.handle, ctypes.byref(o), n, p, r, M.nnz, *at, None, ctypes.byref(nd),
        ctypes.byref(ni), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    count = ctx.launch_count() - before
    ctx.close()
    return count


def test_order_is_read_where_it_counts():
    """The rows' order matters to the copy by tiles and to the blocked passes
    alone: entries too few for both cost no pass over the indices.  The blocked
    passes' plan is four launches."""
    assert _launches(700, 1500, 20, 0.2) == _launches(700, 1500, 20, 0.004) + 1 + 4


# Small factor rows are gathered as fast as they are read from shared memory;
# a line's entries in a block have to pay for the segment.
@pytest.mark.parametrize("n,p,r,density,method,blocked", [
    (300, 500, 2, 0.9, "brunet", False), (300, 500, 4, 0.9, "lee", False),
    (300, 500, 6, 0.9, "brunet", False), (300, 500, 10, 0.9, "lee", False),
    (300, 500, 10, 0.9, "brunet", True), (300, 300, 8, 0.53, "brunet", False),
    (300, 300, 8, 0.53, "lee", True), (700, 1000, 20, 0.03, "lee", False),
    (700, 1000, 20, 0.03, "brunet", True), (700, 700, 32, 0.02, "lee", False),
    (700, 700, 32, 0.03, "lee", True)])
def test_which_passes(n, p, r, density, method, blocked):
    assert _launches(n, p, r, density, method) == _launches(n, p, r, 0.001, method) + 5 * blocked


# The copy by tiles takes 2^23 entries and four a column of a tile: one row and
# a few columns past whole tiles; nearly full ones; rows of one tile; one tile
# of columns.
@pytest.mark.parametrize("n,p,density", [(2177, 8195, 0.5), (3000, 3300, 0.9), (100, 100001, 0.9),
                                         (70001, 300, 0.41)])
def test_csc_by_tiles(oracle, n, p, density):
    V, W0, H0 = _inputs(n, p, 3, density, n + p)
    assert np.count_nonzero(V) > 1 << 23
    _check(oracle, "lee", V, W0, H0, iters=2)


@pytest.mark.parametrize("n,p,density,tiles", [
    (2177, 8195, 0.5, True), (2177, 7000, 0.5, False),  # 8.9 and 7.6 10^6 entries
    (12800, 30000, 0.035, True), (12800, 30000, 0.028, False)])  # 4.5 and 3.6 a tile's column
def test_csc_rule(n, p, density, tiles):
    """By tiles, and after the order, five launches and one; by the sort five."""
    gen = np.random.default_rng(1)
    M = sp.random(n, p, density, "csr", rng=gen)
    assert _launches_of(M, 2, "lee") == _launches(300, 200, 2, 0.5) + tiles
