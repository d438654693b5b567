"""The unbounded nearest-triangle search (SDFGPU_MODE_UNBOUNDED) at the sizes and shapes where its
stages can go wrong, every node against the FP64 oracle, bit for bit: meshes around the number of
triangles queued whole (4), tested at once (32) and kept per node (16); needles, triangles without
area, vertices of high valence; nodes equally far from thousands of triangles (the spilled queue, the
FP64 re-search); grids of one node, one row and ragged edges in every brick shape; meshes far from
the coordinate origin."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu


def check(ctx, X, F, origin, h, N):
    X = np.ascontiguousarray(X, np.float64)
    F = np.ascontiguousarray(F, np.int64)
    N = np.asarray(N, np.int64)
    ctx.set_mesh(X, F)
    d, xp = ctx.distances(origin, h, N, 2, want_xp=True)
    ref, _, _ = oracle.distances(X, F, origin, h, N, mode=2)
    bad = np.flatnonzero(d != ref)
    assert bad.size == 0, f"{bad.size} of {d.size} distances differ, first {bad[:4]}: {d[bad[:4]]} vs {ref[bad[:4]]}"
    # the closest point is one: its distance from the node is the result (to the rounding of a few FP64 steps)
    k, j, i = np.unravel_index(np.arange(d.size), (N + 1)[::-1])
    P = np.asarray(origin) + h * np.stack([i, j, k], 1)
    assert np.allclose(np.linalg.norm(P - xp, axis=1), d, rtol=1e-12, atol=1e-12)


def box_grid(X, n, margin=0.3):
    lo, hi = X.min(0), X.max(0)
    ext = float((hi - lo).max()) * (1 + 2 * margin)
    return 0.5 * (lo + hi) - 0.5 * ext, ext / n, np.array([n, n, n])


@pytest.mark.parametrize("nel", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33, 63, 65, 129])
def test_small_triangle_soups(gpu_ctx, nel):
    rng = np.random.default_rng(nel)
    X = rng.uniform(-1, 1, (nel, 1, 3)) + rng.normal(0, 0.3, (nel, 3, 3))
    o, h, N = box_grid(X.reshape(-1, 3), 17)
    check(gpu_ctx, X.reshape(-1, 3), 1 + np.arange(3 * nel).reshape(-1, 3), o, h, N)


@pytest.mark.parametrize("kind", ["needles", "slivers", "points", "segments", "mixed"])
def test_thin_and_degenerate_triangles(gpu_ctx, kind):
    rng = np.random.default_rng(7)
    n = 120
    a, u, v = rng.uniform(-1, 1, (n, 3)), rng.normal(0, 0.4, (n, 3)), rng.normal(0, 0.4, (n, 3))
    thin = {"needles": 1e-5, "slivers": 1e-9, "points": 0.0, "segments": 0.0, "mixed": 0.0}[kind]
    b = a + u * (0.0 if kind == "points" else 1.0)
    c = a + u * (0.0 if kind == "points" else rng.uniform(0, 1.3, (n, 1))) + thin * v
    if kind == "mixed":  # a closed-looking cloud of ordinary triangles, needles, segments and points
        c[::4] = (a + v)[::4]
        c[1::4] += 1e-6 * v[1::4]
        b[3::4] = a[3::4]
        c[3::4] = a[3::4]
    X = np.stack([a, b, c], 1).reshape(-1, 3)
    o, h, N = box_grid(X, 15)
    # a triangle without area has NaN or undefined normals in the reference; its step is still the
    # oracle's, which the GPU replays
    X32 = X.astype(np.float32).astype(np.float64)
    F = 1 + np.arange(3 * n).reshape(-1, 3)
    gpu_ctx.set_mesh(X32, F)
    d, _ = gpu_ctx.distances(o, h, N, 2)
    ref, _, _ = oracle.distances(X32, F, o, h, N, mode=2)
    bad = np.flatnonzero(d != ref)
    assert bad.size == 0, f"{bad.size} of {d.size} differ, first {bad[:4]}: {d[bad[:4]]} vs {ref[bad[:4]]}"


@pytest.mark.parametrize("valence", [5, 16, 17, 40])
def test_high_valence_apex(gpu_ctx, valence):
    t = 2 * np.pi * np.arange(valence) / valence
    ring = np.stack([np.cos(t), np.sin(t), np.zeros(valence)], 1)
    X = np.concatenate([ring, [[0, 0, 1.0]], [[0, 0, -1.0]]])
    i, j = 1 + np.arange(valence), 1 + (np.arange(valence) + 1) % valence
    F = np.concatenate([np.stack([i, j, np.full(valence, valence + 1)], 1),
                        np.stack([j, i, np.full(valence, valence + 2)], 1)])
    o, h, N = box_grid(X, 20, 0.6)
    check(gpu_ctx, X, F, o, h, N)


@pytest.mark.parametrize("jitter", [0.0, 1e-7, 0.01])
def test_nodes_equally_far_from_all_triangles(gpu_ctx, jitter):
    # the even grid puts a node exactly at the sphere's centre and a brick around it
    V, F = synthetic.icosphere(5, jitter=jitter, seed=3)
    check(gpu_ctx, V, F, np.full(3, -1.2), 0.1, [24, 24, 24])


@pytest.mark.parametrize("N", [(0, 0, 0), (40, 0, 0), (0, 37, 0), (0, 0, 33), (5, 2, 3), (31, 7, 1), (9, 10, 11)])
@pytest.mark.parametrize("brick", [(4, 2, 4), (32, 1, 1), (1, 1, 32), (2, 16, 1), (8, 4, 1)])
def test_ragged_grids_and_brick_shapes(gpu_ctx, N, brick):
    V, F = synthetic.torus(nu=40, nv=18, seed=5)
    gpu_ctx.set_brick(brick)
    try:
        check(gpu_ctx, V, F, np.array([-1.4, -1.3, -0.5]), 0.083, N)
    finally:
        gpu_ctx.set_brick((4, 2, 4))


@pytest.mark.parametrize("shift,scale", [(0.0, 1e-3), (30.0, 1.0), (1e4, 1.0), (-1e6, 50.0)])
def test_mesh_away_from_the_origin(gpu_ctx, shift, scale):
    V, F = synthetic.icosphere(3, jitter=0.02, seed=9)
    X = V * scale + shift
    o, h, N = box_grid(X, 18)
    check(gpu_ctx, X, F, o, h, N)


@pytest.mark.parametrize("kind", ["sphere", "fan", "soup", "one", "repeated"])
@pytest.mark.parametrize("want_xp", [False, True])
def test_three_nearest_vertices(gpu_ctx, kind, want_xp):
    """The reference rule's fallback where every node or most of them take it: meshes coarse against the
    cell, a vertex of 40 triangles, disjoint triangles, fewer than three distinct vertices."""
    rng = np.random.default_rng(11)
    if kind == "sphere":
        X, F = synthetic.icosphere(2, jitter=0.02, seed=4)
    elif kind == "fan":
        t = 2 * np.pi * np.arange(40) / 40
        X = np.concatenate([np.stack([np.cos(t), np.sin(t), 0.2 * np.cos(3 * t)], 1), [[0.1, 0, 0.5]]])
        F = np.stack([1 + np.arange(40), 1 + (np.arange(40) + 1) % 40, np.full(40, 41)], 1)
    elif kind == "soup":
        X, F = rng.uniform(-1, 1, (3 * 37, 3)), 1 + np.arange(3 * 37).reshape(-1, 3)
    elif kind == "one":
        X, F = rng.uniform(-1, 1, (3, 3)), np.array([[1, 2, 3]])
    else:
        X, F = rng.uniform(-1, 1, (3, 3)), np.array([[1, 2, 2], [2, 1, 1]])
    F = np.ascontiguousarray(F, np.int64)
    o, h, N = box_grid(X, 21)
    gpu_ctx.set_mesh(X, F)
    d, xp = gpu_ctx.distances(o, h, N, 0, want_xp=want_xp)
    ref, xpr, _ = oracle.distances(X, F, o, h, N, mode=0, want_xp=want_xp)
    assert np.array_equal(d, ref)
    if want_xp:
        assert np.array_equal(xp, xpr)
