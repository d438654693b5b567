"""The clamped distances (reference rule and true minimum) of meshes whose triangles are small against
the cell, every node against the FP64 oracle, bit for bit: cell sizes from the largest the scatter takes
(vertices at 1.5 or 4 cells from their centroid) to many triangles per cell; spiky surfaces, where the
nearest feature is often a vertex and the reference's vertex-skip rule depends on the triangles' order;
soups of separate triangles; a few triangles without area or unfit for FP32 decisions; z-slabs."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu


def rho_of(X, F):
    T = X[F - 1]
    return np.linalg.norm(T - T.mean(1, keepdims=True), axis=2).max()


def check(ctx, X, F, h, mode):
    X, F = np.ascontiguousarray(X, np.float64), np.ascontiguousarray(F, np.int64)
    lo, hi = X.min(0), X.max(0)
    N = np.minimum(np.ceil((hi - lo) / h).astype(np.int64) + 6, 70)
    o = 0.5 * (lo + hi) - 0.5 * h * N + 0.123 * h
    ctx.set_mesh(X, F)
    d, _ = ctx.distances(o, h, N, mode)
    ref, _, _ = oracle.distances(X, F, o, h, N, mode=mode)
    bad = np.flatnonzero(d != ref)
    assert bad.size == 0, f"{bad.size} of {d.size} distances differ, first {bad[:4]}: {d[bad[:4]]} vs {ref[bad[:4]]}"
    assert (ref < h).any()
    return ctx.stats()


MODES = [0, 1]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("level,jitter", [(0, 0.0), (1, 0.3), (2, 0.0), (2, 0.25), (3, 0.1), (4, 0.02), (5, 0.3)])
@pytest.mark.parametrize("cells", [0.03, 0.3, 0.66, 1.49])
def test_spheres(gpu_ctx, level, jitter, cells, mode):
    V, F = synthetic.icosphere(level, jitter=jitter, seed=level)
    st = check(gpu_ctx, V, F, rho_of(V, F) / cells, mode)
    assert st["band_nodes"] > 0  # the scatter took it


@pytest.mark.parametrize("cells", [2.0, 3.9, 4.2])
def test_true_minimum_with_larger_triangles(gpu_ctx, cells):
    V, F = synthetic.icosphere(2, jitter=0.1, seed=8)
    st = check(gpu_ctx, V, F, rho_of(V, F) / cells, 1)
    assert (st["band_nodes"] > 0) == (cells < 4.0)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("nel", [1, 2, 31, 127, 128, 129, 1000])
def test_soups(gpu_ctx, nel, mode):
    rng = np.random.default_rng(nel)
    X = (rng.uniform(-1, 1, (nel, 1, 3)) + rng.normal(0, 0.05, (nel, 3, 3))).reshape(-1, 3)
    F = 1 + np.arange(3 * nel).reshape(-1, 3)
    check(gpu_ctx, X, F, max(rho_of(X, F) / 1.2, 0.05), mode)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("cells", [0.2, 0.9])
def test_few_unfit_triangles(gpu_ctx, mode, cells):
    """Needles, segments and points on an ordinary surface (under one triangle in 64): the nodes nearest to
    them replay the whole fold."""
    V, F = synthetic.icosphere(4, jitter=0.05, seed=6)
    rng = np.random.default_rng(2)
    at = rng.choice(len(F), 60, replace=False)
    extra, X = [], [V]
    n = len(V)
    for k, t in enumerate(at):
        a, b, c = V[F[t] - 1]
        a, b, c = 1.02 * a, 1.02 * b, 1.02 * c
        if k % 3 == 0:
            c = a + (b - a) * 0.4 + 1e-7
        elif k % 3 == 1:
            c = b
        else:
            b = c = a
        X.append(np.stack([a, b, c]))
        extra.append([n + 1, n + 2, n + 3])
        n += 3
    X = np.concatenate(X)
    F2 = np.concatenate([F, np.array(extra)])
    st = check(gpu_ctx, X, F2, rho_of(X, F2) / cells, mode)
    assert st["band_nodes"] > 0


@pytest.mark.parametrize("mode", MODES)
def test_slab_and_signed(gpu_ctx, mode):
    V, F = synthetic.torus(nu=96, nv=40, seed=4)
    h = 0.06
    N = np.array([45, 44, 13])
    o = np.array([-1.35, -1.33, -0.41])
    gpu_ctx.set_mesh(V, F)
    full = gpu_ctx.sdf(o, h, N, mode)
    n = int((N[0] + 1) * (N[1] + 1))
    for k0, k1 in ((0, 0), (3, 8), (13, 13)):
        part = gpu_ctx.sdf_slab(o, h, N, k0, k1, mode)
        assert np.array_equal(part, full[n * k0:n * (k1 + 1)])


@pytest.mark.parametrize("n", [3, 5, 7, 9, 16])
@pytest.mark.parametrize("drop", [1, 40, 200])
def test_adaptive_rays_of_few_and_many_nodes(gpu_ctx, n, drop):
    """An open surface on growing grids: the undecided nodes' rays go against all triangles while they are
    few and through the LBVH beyond; signs and confidences equal the oracle's either way."""
    V, F = synthetic.icosphere(3, jitter=0.05, seed=7)
    F = np.ascontiguousarray(np.delete(F, np.random.default_rng(n).choice(len(F), drop, replace=False), axis=0))
    o, h, N = np.full(3, -1.21), 2.37 / n, np.array([n, n, n])
    gpu_ctx.set_mesh(V, F)
    s, c = gpu_ctx.signs(o, h, N)
    ref = oracle.signs(V, F, o, h, N)
    assert np.array_equal(s, ref["sign"]) and np.array_equal(c, ref["conf"])


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("size", [0.1, 0.6, 1.4])
@pytest.mark.parametrize("cones", [40, 4000])
def test_separate_cones(gpu_ctx, cones, size, mode):
    """Open cones whose apex is the nearest point of most nodes around them, the case that replays the
    reference's fold: a few such nodes, and more than fit the fixed places of their candidate lists."""
    rng = np.random.default_rng(cones)
    a = rng.uniform(0, 1, (cones, 1, 3))
    ring = a + size / 66.0 * rng.normal(0, 0.3, (cones, 3, 3)) + size / 66.0 * rng.normal(0, 0.5, (cones, 1, 3))
    X = np.concatenate([a, ring], 1).reshape(-1, 3)
    b = 4 * np.arange(cones)[:, None] + 1
    F = np.concatenate([b + np.array([[0, 1, 2]]), b + np.array([[0, 2, 3]]), b + np.array([[0, 3, 1]])], 0)
    check(gpu_ctx, X, F, 1.0 / 64.0, mode)
