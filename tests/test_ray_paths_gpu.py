"""The adaptive rays of open surfaces on either side of the number of undecided nodes up to which they test every
triangle (24) and beyond which they walk the LBVH: signs and confidences of every node against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu

ALL_PAIRS = 24


def test_both_sides(gpu_ctx):
    few = many = 0
    for n in range(3, 15):
        for drop in (1, 3, 12, 60):
            V, F = synthetic.icosphere(3, jitter=0.05, seed=n)
            F = np.ascontiguousarray(np.delete(F, np.random.default_rng(drop).choice(len(F), drop, replace=False), axis=0))
            o, h, N = np.full(3, -1.21), 2.37 / n, np.array([n, n, n])
            gpu_ctx.set_mesh(V, F)
            s, c = gpu_ctx.signs(o, h, N)
            undecided = gpu_ctx.stats()["undecided_nodes"]
            ref = oracle.signs(V, F, o, h, N)
            assert np.array_equal(s, ref["sign"]) and np.array_equal(c, ref["conf"])
            few += 0 < undecided <= ALL_PAIRS
            many += undecided > ALL_PAIRS
    assert few > 5 and many > 5
