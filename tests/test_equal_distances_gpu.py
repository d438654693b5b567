"""Nodes that lie equally far from several triangles, up to a few roundings: every node of grids placed
symmetrically about boxes, against the FP64 oracle, bit for bit.  Which of the nearly equal values the reference
takes depends on the triangles' order and on the box test that starts each step."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("pieces", [1, 2, 4])  # the faces' quads along each axis: large and small triangles
def test_symmetric_grids_about_boxes(gpu_ctx, pieces, mode):
    bad = []
    for seed in range(150):
        rng = np.random.default_rng(seed)
        lo, hi = -rng.integers(1, 5, 3) / 8.0, rng.integers(1, 5, 3) / 8.0
        V, F = synthetic.box(tuple(lo), tuple(hi))
        for _ in range(pieces // 2):  # midpoint subdivision
            T = V[F - 1]
            a, b, c = T[:, 0], T[:, 1], T[:, 2]
            p, q, r = 0.5 * (a + b), 0.5 * (b + c), 0.5 * (c + a)
            S = np.stack([np.stack(t, 1) for t in ((a, p, r), (p, b, q), (r, q, c), (p, q, r))], 1).reshape(-1, 3)
            V, inv = np.unique(S, axis=0, return_inverse=True)
            F = 1 + inv.reshape(-1, 3)
        scale = 1.0 if seed % 3 == 0 else 10.0 ** rng.uniform(-4, 4)
        V = V * scale
        lo, hi = V.min(0), V.max(0)
        h = (hi - lo).max() / (float(rng.choice([4, 8, 16])) if seed % 2 else rng.uniform(4, 20))
        N = np.minimum(np.ceil((hi - lo) / h).astype(np.int64) + rng.integers(0, 6), 24)
        o = 0.5 * (lo + hi) - 0.5 * h * N
        gpu_ctx.set_mesh(V, F)
        d, _ = gpu_ctx.distances(o, h, N, mode)
        ref, _, _ = oracle.distances(V, F, o, h, N, mode=mode)
        if not np.array_equal(d, ref):
            bad.append((seed, int((d != ref).sum()), float(np.abs(d - ref).max() / h)))
    assert not bad


@pytest.mark.parametrize("level,copies", [(0, 1), (1, 1), (2, 1), (3, 1), (0, 17), (1, 5), (2, 20)])
def test_closest_points_of_more_ties_than_a_node_keeps(gpu_ctx, level, copies):
    """The centre of a sphere, and the nodes around meshes of coincident triangles: the lowest index has it."""
    V, F = synthetic.icosphere(level, jitter=0.0 if copies == 1 else 0.1, seed=level)
    F = np.repeat(F, copies, axis=0)[np.random.default_rng(copies).permutation(copies * len(F))]
    N = np.array([12, 12, 12])
    gpu_ctx.set_mesh(V, F)
    d, x = gpu_ctx.distances(np.full(3, -1.5), 0.25, N, 2, want_xp=True)
    ref, xr, _ = oracle.distances(V, F, np.full(3, -1.5), 0.25, N, mode=2, want_xp=True)
    assert np.array_equal(d, ref) and np.array_equal(x, xr)
