"""A batch large enough for four columns a thread (f32) gives each solve the
bits it has in a batch small enough for two: the same operations column by
column.  Ranks of every bucket; odd lengths."""
from __future__ import annotations

import numpy as np
import pytest

from nmf_rs import consensus

pytestmark = pytest.mark.gpu


def test_column_widths_agree():
    gen = np.random.default_rng(5)
    n, p = 517, 531  # two 512-column tiles a step
    V = gen.gamma(0.5, 1.0, (n, 6)) @ gen.gamma(0.5, 1.0, (6, p))
    V[gen.random((n, p)) < 0.3] = 0.0
    # 600 groups of one solve: 600 * 2 * 4 warps of four columns, above the
    # 32 a multiprocessor that a step needs to take them
    ranks = [16, 9, 7, 11, 10, 8] * 100
    starts = [(gen.random((n, r)), gen.random((r, p))) for r in ranks]
    wide = consensus.run_batch(V, starts, 11, precision="fp32")
    narrow = consensus.run_batch(V, starts[:6], 11, precision="fp32")
    for (W, H), (W2, H2) in zip(narrow, wide):
        np.testing.assert_array_equal(W, W2)
        np.testing.assert_array_equal(H, H2)


def test_one_bucket_widths_agree():
    """Ranks of one bucket take two columns a thread only within the waves of
    four, and never above rank 14: alone or many, a solve has the bits it has
    beside ranks of every bucket."""
    gen = np.random.default_rng(6)
    n, p = 517, 531
    V = gen.gamma(0.5, 1.0, (n, 6)) @ gen.gamma(0.5, 1.0, (6, p))
    V[gen.random((n, p)) < 0.3] = 0.0
    ranks = [16, 15, 14, 10, 9, 8, 3]
    starts = [(gen.random((n, r)), gen.random((r, p))) for r in ranks]
    mixed = consensus.run_batch(V, starts, 11, precision="fp32")
    for start, (W, H) in zip(starts, mixed):
        for many in (1, 200):  # 200: two waves and more of two columns, not of four
            got = consensus.run_batch(V, [start] * many, 11, precision="fp32")
            np.testing.assert_array_equal(got[-1][0], W)
            np.testing.assert_array_equal(got[-1][1], H)
