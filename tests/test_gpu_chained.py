"""Chained launches: from the second iteration a run's kernels may start
before the one ahead of them has drained.  With the per-kernel timing on they
are launched plainly, each after the last; the same kernels on the same data
must give the same bits, whatever overlaps: few and many factor tiles, every
kernel that can stand between two steps, and a stop in mid-run."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import nmf_rs
from nmf_rs import _native, synthetic

pytestmark = pytest.mark.gpu


def _run(method, V, W0, H0, iters, precision, stop, timing):
    n, p = V.shape
    Vd, Wd, Hd = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (V, W0, H0))
    o = _native.default_options()
    o.method = _native.parse_method(method)
    o.stop = stop
    o.max_iter = iters
    o.precision = _native.PRECISIONS[precision]
    o.stationary_th = 1e-3 * float(V.sum())
    o.device = 0
    dev = torch.zeros(iters + 1, dtype=torch.float64, device="cuda")
    ctx = _native.Context(0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    try:
        ctx.set_timing(timing)
        res = ctx.run(o, n, p, W0.shape[1], Vd.data_ptr(), _native.F64, p, Wd.data_ptr(),
                      Hd.data_ptr(), dev_ptr=dev.data_ptr(), stream=side.cuda_stream)
        torch.cuda.synchronize()
        return Wd.cpu().numpy(), Hd.cpu().numpy(), dev.cpu().numpy(), res
    finally:
        ctx.close()


@pytest.mark.parametrize("stop", [0, 1])
@pytest.mark.parametrize("method,precision", [
    ("brunet", "fp64"), ("lee", "fp64"), ("hals", "fp64"), ("ehals", "fp64"), ("dnmf", "fp64"),
    ("nsNMF", "fp64"), ("brunet", "fp32"), ("lee", "fp32"), ("lee", "bf16x3"),
    ("brunet", "bf16x3")])
@pytest.mark.parametrize("n,p", [(33, 70), (210, 10100), (9700, 150)])
def test_chained_equals_plain(n, p, method, precision, stop):
    V = synthetic.counts_matrix(n, p, 5, 0.3, seed=n)
    W0, H0 = nmf_rs.random_init(V, 6, seed=4)
    got = _run(method, V, W0, H0, 57, precision, stop, False)
    want = _run(method, V, W0, H0, 57, precision, stop, True)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    np.testing.assert_array_equal(got[2], want[2])
    assert got[3] == want[3]
