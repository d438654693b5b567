"""Signs from the hits of the grid's rows, every node against the FP64 oracle: grids whose node counts lie
around the 32 nodes of a mask word and the 4 x 4 columns of a vote tile; nodes exactly on the surface and
rows exactly through edges and vertices (hits that merge); surfaces a few rounding errors or a few times
the merge distance apart; rows with more hits than a node sorts; meshes that reach past the grid; slabs."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu


def boxes(bounds):
    Vs, Fs, n = [], [], 0
    for lo, hi in bounds:
        V, F = synthetic.box(lo, hi)
        Vs.append(V)
        Fs.append(F + n)
        n += len(V)
    return np.concatenate(Vs), np.concatenate(Fs)


def check(ctx, X, F, o, h, N, **kw):
    X, F = np.ascontiguousarray(X, np.float64), np.ascontiguousarray(F, np.int64)
    o, N = np.asarray(o, np.float64), np.asarray(N, np.int64)
    ctx.set_mesh(X, F)
    s, c = ctx.signs(o, h, N, **kw)
    ref = oracle.signs(X, F, o, h, N, **kw)
    # a node on the surface has a winding number of 0.5 to the last bit of atan2, in either arithmetic
    # (the library counts these nodes as ambiguous); every other sign is compared
    tie = (ref["fallback"] != 0) & (np.abs(np.abs(ref["winding"]) - 0.5) < 1e-9)
    assert np.array_equal(s[~tie], ref["sign"][~tie])
    assert np.array_equal(c, ref["conf"])
    return ctx.stats()


@pytest.mark.parametrize("n", [(31, 3, 2), (32, 4, 4), (33, 5, 3), (64, 1, 9), (3, 33, 32), (2, 4, 65), (1, 1, 1), (97, 2, 34)])
def test_ragged(gpu_ctx, n):
    V, F = synthetic.icosphere(2, jitter=0.2, seed=3)
    h = 2.4 / max(n)
    o = -0.5 * h * (np.array(n) - 1.0) + 0.01
    check(gpu_ctx, V, F, o, h, np.array(n) - 1)


@pytest.mark.parametrize("off", [0.0, 1e-9, 0.5e-8, 1e-8, 1.5e-8, 1e-5, 0.03125])
@pytest.mark.parametrize("rays", [dict(), dict(min_rays=4, max_rays=12), dict(use_winding_fallback=False, confidence_threshold=0.9)])
def test_nodes_on_the_surface(gpu_ctx, off, rays):
    X, F = boxes([((0.25, 0.25, 0.25), (0.75, 1.0, 0.5))])  # faces, edges and diagonals on the nodes
    check(gpu_ctx, X, F, np.array([0.0, 0.0, 0.0]) + off, 0.0625, (16, 19, 12), **rays)


@pytest.mark.parametrize("gap", [0.0, 1e-12, 2.4e-9, 2.6e-9, 9.99999999e-9, 1e-8, 1.00000001e-8, 3e-8, 1e-6])
def test_surfaces_close_together(gpu_ctx, gap):
    X, F = boxes([((0.2, 0.2, 0.2), (0.8, 0.8, 0.8))] + [((0.2 + g, 0.2 + g, 0.2 + g), (0.8 - g, 0.8 - g, 0.8 - g))
                                                        for g in (gap, 2.0 * gap, 3.0 * gap)])
    check(gpu_ctx, X, F, (0.013, 0.021, 0.007), 0.0625, (15, 14, 16))


@pytest.mark.parametrize("layers", [30, 31, 32, 33, 40])
def test_many_hits_in_a_row(gpu_ctx, layers):
    t = 0.4 * np.arange(layers) / layers
    X, F = boxes([((q, q, q), (1.0 - q, 1.0 - q, 1.0 - q)) for q in t])
    st = check(gpu_ctx, X, F, (-0.0531, 0.0117, 0.0213), 0.0625, (16, 15, 14))
    assert st["row_hits"] > 0


@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (1e-3, 0.0), (50.0, 0.0), (1.0, 1e4), (1.0, -3e6)])
def test_open_surface_past_the_grid(gpu_ctx, scale, shift):
    V, F = synthetic.icosphere(3, jitter=0.1, seed=5)
    V, F = V * scale + shift, F[: len(F) * 7 // 8]  # rays through the hole disagree
    h = scale * 0.06
    st = check(gpu_ctx, V, F, np.array([-0.4, -0.3, -0.5]) * scale + shift, h, (18, 21, 13))
    assert st["undecided_nodes"] > 0


def test_slabs(gpu_ctx):
    X, F = boxes([((0.25, 0.25, 0.25), (0.75, 1.0, 0.5)), ((0.1, 0.3, 0.2), (0.9, 0.6, 1.1))])
    o, h, N = np.array([0.0, 0.0, 0.0]), 0.0625, np.array([16, 19, 20], np.int64)
    gpu_ctx.set_mesh(X, F)
    whole = gpu_ctx.sdf(o, h, N)
    plane = int((N[0] + 1) * (N[1] + 1))
    for k0, k1 in [(0, 0), (1, 5), (6, 20)]:
        assert np.array_equal(gpu_ctx.sdf_slab(o, h, N, k0, k1), whole[k0 * plane:(k1 + 1) * plane])


@pytest.mark.parametrize("nel", [12, 36, 96, 120])
@pytest.mark.parametrize("nodes", [12, 40, 97])
def test_triangles_over_many_rows(gpu_ctx, nel, nodes):
    """Few triangles, each across up to nodes^2 rows, so that several threads and blocks share one."""
    rng = np.random.default_rng(nel)
    X, F = boxes([(lo, lo + rng.uniform(0.2, 0.6, 3)) for lo in rng.uniform(0.0, 0.4, (nel // 12, 3))])
    st = check(gpu_ctx, X, F, (-0.011, -0.017, -0.013), 1.1 / nodes, (nodes, nodes - 3, nodes // 2))
    assert st["row_hits"] > 0
