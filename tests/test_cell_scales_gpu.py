"""Every distance mode at the ends of the range of cell sizes, every node against the FP64 oracle, bit for bit.
Around 1e10, the reference's initial minimum (abs(-1.0e10), src/SignedDistances/dfOnTriangularMesh.jl:31): above
it a node that no triangle comes closer to keeps that minimum, whether or not it has candidates.  And where
the squares of FP32 distances, or the tile fold's products of four lengths, overflow or lose digits by
underflow."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu



def check(ctx, h, cells, mode, want_xp, away=0.0, level=3, copies=1):
    """A sphere whose triangles reach `cells` cells from their centroids, `away` radii from the origin."""
    V, F = synthetic.icosphere(level, jitter=0.1, seed=5)
    F = np.repeat(F, copies, axis=0)
    T = V[F - 1]
    V = V * (cells * h / np.linalg.norm(T - T.mean(1, keepdims=True), axis=2).max())
    V = V + away * V.max()
    lo, hi = V.min(0), V.max(0)
    N = np.minimum(np.ceil((hi - lo) / h).astype(np.int64) + 14, 40)
    o = 0.5 * (lo + hi) - 0.5 * h * N + 0.123 * h
    ctx.set_mesh(V, F)
    ref, _, _ = oracle.distances(V, F, o, h, N, mode=mode)
    d, _ = ctx.distances(o, h, N, mode, want_xp=want_xp)
    assert np.array_equal(d, ref)
    return ctx.stats()


H = [5e9, 1e10, 1.0000000001e10, 3e10, 1e12]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", H)
@pytest.mark.parametrize("cells", [0.01, 0.4, 1.4])
def test_scatter(gpu_ctx, h, cells, mode):
    assert check(gpu_ctx, h, cells, mode, False)["band_nodes"] > 0


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", H)
@pytest.mark.parametrize("away", [0.0, 100.0])  # the scatter takes meshes near the origin
def test_tiles(gpu_ctx, h, mode, away):
    assert check(gpu_ctx, h, 0.01, mode, away == 0.0, away)["band_nodes"] == 0


@pytest.mark.parametrize("h", H)
def test_unbounded(gpu_ctx, h):
    check(gpu_ctx, h, 0.4, 2, True)


SMALL = [2e-15, 5e-16, 1e-20, 1e-22, 1e-24]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", SMALL)
@pytest.mark.parametrize("cells,level", [(0.3, 4), (0.66, 5), (1.4, 3)])
def test_small_cells(gpu_ctx, h, cells, level, mode):
    st = check(gpu_ctx, h, cells, mode, False, level=level)
    assert (st["band_nodes"] > 0) == (h > 1e-15)  # the scatter takes the larger ones


@pytest.mark.parametrize("mode", [0, 2])  # with closest points: the nearest-vertex fallback, the search
@pytest.mark.parametrize("h", SMALL)
@pytest.mark.parametrize("cells,level", [(0.3, 4), (0.66, 5), (1.4, 3)])
def test_searches_of_small_cells(gpu_ctx, h, cells, level, mode):
    check(gpu_ctx, h, cells, mode, True, level=level)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("h", H + [1e8, 1e16, 1e-9, 1e-10, 3e-11, 1e-11, 1e-12])
@pytest.mark.parametrize("cells", [0.4, 2.5, 6.0])
def test_tiles_where_products_of_four_lengths_leave_fp32(gpu_ctx, h, cells, mode):
    check(gpu_ctx, h, cells, mode, True)


@pytest.mark.parametrize("h", [1e8, 1e7, 1e6, 1e5, 1.0, 1e-6, 1e-8, 1e-12, 1e-16])
@pytest.mark.parametrize("cells,level", [(6.0, 1), (8.1, 2)])
def test_large_triangles_off_the_candidates(gpu_ctx, h, cells, level):
    """The nodes within a cell of a triangle whose centroid is far take the nearest-vertex fallback."""
    assert check(gpu_ctx, h, cells, 0, False, level=level)["knn_fallback_nodes"] > 0


@pytest.mark.parametrize("h", [1e8, 1e7, 1e6, 1e5, 1.0, 1e-6, 1e-8, 1e-12, 1e-16])
def test_more_coincident_triangles_than_a_node_keeps(gpu_ctx, h):
    check(gpu_ctx, h, 6.0, 2, True, level=0, copies=20)
