"""Meshes 1e7 to 2e10 of their sizes from the coordinate origin, where a coordinate's rounding is a visible part of a
cell, with grid rows along their borders: distances, signs and confidences of every node against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("away", [1e7, 3e8, 3e9, 2e10])
@pytest.mark.parametrize("kind", ["plane", "box"])
def test_rows_along_the_border(gpu_ctx, kind, away):
    for seed in range(40):
        rng = np.random.default_rng(seed)
        if kind == "plane":
            m = int(rng.integers(2, 12))
            x, y = np.meshgrid(np.arange(m), np.arange(m), indexing="ij")
            V = np.stack([x.ravel() / (m - 1.0), y.ravel() / (m - 1.0), 0.0 * x.ravel()], 1)
            i = (np.arange(m - 1)[:, None] * m + np.arange(m - 1)[None]).ravel() + 1
            F = np.concatenate([np.stack([i, i + m, i + m + 1], 1), np.stack([i, i + m + 1, i + 1], 1)])
        else:
            V, F = synthetic.box((0.0, 0.0, 0.0), tuple(rng.integers(1, 5, 3) / 4.0))
        V = V + away * rng.normal(size=3)
        lo, hi = V.min(0), V.max(0)
        h = float((hi - lo).max()) / int(rng.integers(3, 12))
        N = np.ceil((hi - lo) / h).astype(np.int64) + 2
        o = lo - (0.0 if seed % 2 else h)
        gpu_ctx.set_mesh(V, F)
        s, c = gpu_ctx.signs(o, h, N)
        ref = oracle.signs(V, F, o, h, N)
        tie = (ref["fallback"] != 0) & (np.abs(np.abs(ref["winding"]) - 0.5) < 1e-9)
        assert np.array_equal(c, ref["conf"]), seed
        assert np.array_equal(s[~tie], ref["sign"][~tie]), seed
        for mode in (0, 1, 2):
            d, _ = gpu_ctx.distances(o, h, N, mode)
            assert np.array_equal(d, oracle.distances(V, F, o, h, N, mode=mode)[0]), (seed, mode)
