"""The clamped distances of meshes whose nodes replay the reference's fold in the scatter: every triangle more
often than a node has slots, so that all near nodes replay it, from lists in fixed places, in counted places,
or, when the lists do not fit, by scans of a small mesh or through the tile fold; and fans of more triangles than
a list holds.  A sample of the nodes against the FP64 oracle, and where signs can be had all nodes against the
tile fold (which persistent batches take), bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from workloads import synthetic

pytestmark = pytest.mark.gpu

# triangles a node keeps, candidates a list holds, lists with fixed places, triangles of a mesh that is scanned
SLOTS, LIST, FIXED, SCANNED = 16, 1024, 16384, 16384


def check(ctx, X, F, h, mode, signed=True):
    X, F = np.ascontiguousarray(X, np.float64), np.ascontiguousarray(F, np.int64)
    lo, hi = X.min(0), X.max(0)
    N = np.ceil((hi - lo) / h).astype(np.int64) + 6
    o = 0.5 * (lo + hi) - 0.5 * h * N + 0.123 * h
    ctx.set_mesh(X, F)
    d, _ = ctx.distances(o, h, N, mode)
    st = ctx.stats()
    if signed:  # (a ray takes at most 256 hits)
        fold = ctx.sdf_batch([(X, F, o, h, N)], mode, streams=1, autotune=False, persistent=True, want_parts=True)[0][1]
        sdf, dist, sign, _ = ctx.sdf(o, h, N, mode, want_parts=True)
        assert np.array_equal(d, fold) and np.array_equal(dist, fold) and np.array_equal(sdf, fold * sign)
    near = np.flatnonzero(d < h)
    nodes = np.sort(np.random.default_rng(1).choice(d.size, min(4000, d.size), replace=False))
    nodes = np.union1d(nodes, near[::97])
    ref, _, _ = oracle.distances(X, F, o, h, N, mode=mode, nodes=nodes)
    assert np.array_equal(d[nodes], ref)
    return st, near.size


def sphere(level, copies, cells=0.85):
    """An icosphere of radius 1, each triangle `copies` times, and a cell size of which its triangles reach
    `cells`: at 0.85 about 25 of its triangles lie within a near node's bound, at 1.2 about 13."""
    V, F = synthetic.icosphere(level, jitter=0.002, seed=3)
    T = V[F - 1]
    return V, np.repeat(F, copies, axis=0), np.linalg.norm(T - T.mean(1, keepdims=True), axis=2).max() / cells


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("level,copies,cells,lists", [
    (4, SLOTS + 1, 0.85, "fixed"), (5, SLOTS + 1, 0.85, "counted"),  # 12M candidates for 16M places
    (5, 3 * SLOTS, 1.2, "none"),                                     # 32M candidates, 800 a node
    (4, 4 * SLOTS, 0.85, "none"),                                    # 1600 a node
    (2, 12 * SLOTS, 0.85, "scan")])                                  # 4800 a node, 61k triangles
def test_every_near_node_replays(gpu_ctx, level, copies, cells, lists, mode):
    V, F, h = sphere(level, copies, cells)
    if lists == "scan":
        F = F[:SCANNED]
    st, near = check(gpu_ctx, V, F, h, mode, level == 4 or copies < 2 * SLOTS)
    if lists == "none":
        assert st["tile_pairs"] > 0  # the tile fold took the call
    else:
        assert st["tile_pairs"] == 0 and st["band_nodes"] >= near
        assert (near <= FIXED) == (lists != "counted")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("rest", [0, SCANNED])
@pytest.mark.parametrize("fan", [LIST // 2, LIST, LIST + 1, 3 * LIST])
def test_fans(gpu_ctx, fan, rest, mode):
    """Cones whose apex is a vertex of `fan` triangles and the nearest point of the nodes above it, alone and
    beside a mesh too large to be scanned."""
    a = 2.0 * np.pi * np.arange(fan) / fan
    X = np.concatenate([[[0.0, 0.0, 1.0]], np.stack([0.15 * np.cos(a), 0.15 * np.sin(a), 0.8 + 0.0 * a], 1)])
    i = np.arange(fan)
    F = np.stack([np.ones(fan), 2 + i, 2 + (i + 1) % fan], 1)
    if rest:
        V, G = synthetic.icosphere(5, seed=3)
        X, F = np.concatenate([X, 0.5 * V]), np.concatenate([F, G + len(X)])
    st, _ = check(gpu_ctx, X, F, 0.13, mode, False)
    assert (st["tile_pairs"] > 0) == (fan > LIST and rest > 0)
    assert (st["band_nodes"] > 0) == (st["tile_pairs"] == 0)


def test_slabs_that_the_tile_fold_takes_over(gpu_ctx):
    V, F, h = sphere(4, 4 * SLOTS)
    o = V.min(0) - 2.9 * h
    N = np.ceil((V.max(0) - o) / h).astype(np.int64) + 2
    gpu_ctx.set_mesh(V, F)
    whole, dist, sign, _ = gpu_ctx.sdf(o, h, N, 0, want_parts=True)
    assert gpu_ctx.stats()["tile_pairs"] > 0
    n = int((N[0] + 1) * (N[1] + 1))
    for k0, k1 in ((0, 4), (5, 20), (21, int(N[2]))):
        part = gpu_ctx.sdf_slab(o, h, N, k0, k1, 0, want_parts=True)
        for a, b in zip(part, (whole, dist, sign)):
            assert np.array_equal(a, b[n * k0:n * (k1 + 1)])


def test_the_call_after_it(gpu_ctx):
    """A call that the tile fold took over leaves nothing behind for the next one."""
    V, F, h = sphere(4, 4 * SLOTS)
    check(gpu_ctx, V, F, h, 0)
    st, _ = check(gpu_ctx, V, F[::4 * SLOTS], h, 0)
    assert st["tile_pairs"] == 0 and st["band_nodes"] > 0
