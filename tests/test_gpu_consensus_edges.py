"""Edges of the consensus kernels on the GPU: label planes (ranks around the
plane counts, solves around whole words, columns around whole tiles) against
numpy's pair counts, and the average-linkage tree around the sizes where a
thread holds one more entry of a row, up to the sizes whose cluster sizes and
chains leave shared memory."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from nmf_rs import _native, consensus  # noqa: E402


@pytest.mark.parametrize("p", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("rank,nsel", [(1, 1), (2, 31), (3, 32), (4, 33), (9, 64), (16, 65),
                                       (17, 7), (255, 40)])
def test_consensus_matrix_counts(p, rank, nsel):
    gen = np.random.default_rng(100 * rank + p)
    ranks = np.full(nsel + 1, rank, dtype=np.int32)
    H = torch.from_numpy(gen.random((int(ranks.sum()), p))).cuda()
    sel = np.arange(1, nsel + 1, dtype=np.int32)
    out = torch.full((p, p), -1.0, dtype=torch.float32, device="cuda")
    ctx = _native.Context(0)
    _native.check(_native.load().nmfcu_consensus_device(
        ctx.handle, p, nsel + 1, consensus._ranks_ptr(ranks), ctypes.c_void_p(H.data_ptr()), nsel,
        consensus._ranks_ptr(sel), ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    ctx.close()
    Hh = H.cpu().numpy()
    count = np.zeros((p, p), dtype=np.int64)
    for i in sel:
        lab = Hh[i * rank:(i + 1) * rank].argmax(0)
        count += lab[:, None] == lab[None, :]
    # the quotient of two small integers in f32: exact
    np.testing.assert_array_equal(out.cpu().numpy(),
                                  count.astype(np.float32) / np.float32(nsel))


def _weighted_upgma(Dk, w):
    """(heights, pair weights) of the average-linkage tree of k groups of
    sizes w at distances Dk (no ties between groups)."""
    Dk, w = Dk.copy(), list(map(float, w))
    live = list(range(len(w)))
    merges = []
    while len(live) > 1:
        d, a, b = min((Dk[i, j], i, j) for x, i in enumerate(live) for j in live[x + 1:])
        merges.append((d, w[a] * w[b]))
        for i in live:
            if i not in (a, b):
                Dk[i, b] = Dk[b, i] = (w[a] * Dk[i, a] + w[b] * Dk[i, b]) / (w[a] + w[b])
        w[b] += w[a]
        live.remove(a)
    return merges


# 2048 indices a row entry of a thread: 1 to 6 and 8 entries, any number above
# 16384; sizes and chains in global memory above 20480.
@pytest.mark.parametrize("p", [2048, 2049, 4097, 6145, 8193, 10241, 12289, 16384, 16385, 20481])
def test_tree_of_grouped_columns(p):
    """Columns in k groups, identical within a group: the tree joins each
    group at height 0 and then is the small weighted tree of the groups."""
    k = 7
    gen = np.random.default_rng(p)
    lab = gen.integers(0, k, p)
    M = gen.permutation(np.arange(1, k * k + 1)).reshape(k, k) / 64.0
    M = (M + M.T).astype(np.float32) / np.float32(2.0)
    M = np.minimum(M, np.float32(0.99))
    np.fill_diagonal(M, 1.0)
    dM, dl = torch.from_numpy(M).cuda(), torch.from_numpy(lab).cuda()
    C = dM[dl][:, dl].contiguous()
    coph, disp = consensus.consensus_stats(C)
    w = np.bincount(lab, minlength=k)
    D = 1.0 - M.astype(np.float64)
    merges = _weighted_upgma(D, w)
    N = p * (p - 1) / 2
    iu = np.triu_indices(k, 1)
    pw = (w[:, None] * w[None, :])[iu].astype(np.float64)
    zero = N - pw.sum()  # the pairs within groups, at distance 0
    md = (pw * D[iu]).sum() / N
    var_d = (pw * (D[iu] - md) ** 2).sum() + zero * md * md
    h = np.array([m[0] for m in merges])
    n = np.array([m[1] for m in merges])
    mc = (n * h).sum() / N
    cov = (n * (h - mc) * (h - md)).sum() + zero * mc * md
    var_c = (n * (h - mc) ** 2).sum() + zero * mc * mc
    # heights are averages of up to k rounded averages; the sums over p^2
    # pairs round at 1e-16 * sqrt(pairs) at most
    assert coph == pytest.approx(cov / np.sqrt(var_d * var_c), abs=1e-9)
    ww = w[:, None] * w[None, :].astype(np.float64)
    assert disp == pytest.approx((ww * 4.0 * (M.astype(np.float64) - 0.5) ** 2).sum() / p / p,
                                 abs=1e-9)


def test_stats_of_nan_consensus_end():
    """A NaN entry leaves no spread to correlate: 1, as for a constant matrix,
    and the tree ends."""
    C = torch.rand((300, 300), device="cuda")
    C = (C + C.T) / 2
    C[5, :] = float("nan")
    C[:, 5] = float("nan")
    coph, disp = consensus.consensus_stats(C)
    assert coph == 1.0 and np.isnan(disp)
