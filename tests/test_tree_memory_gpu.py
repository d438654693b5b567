"""A mesh whose search tree does not fit the device's memory, after a mesh whose calls used one: the calls that
do not need the tree run, those that do report it, and run once there is memory."""

from __future__ import annotations

import numpy as np
import pytest

from workloads import synthetic

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_a_tree_that_does_not_fit():
    import torch
    from stl2sdf import _native

    V, F = synthetic.icosphere(2, jitter=0.05, seed=1)
    o, h, N = np.full(3, -1.6), 0.1, np.array([32, 32, 12])
    # 2.1M triangles: 1370 MB for the mesh (580 B a triangle and an eighth), 870 MB for its tree (372 B)
    X, IEN = synthetic.torus(nu=1024, nv=1024, seed=1)
    ctx = _native.Context(0)
    try:
        ctx.set_mesh(V, F)
        ctx.distances(o, h, N, 0)  # kernels are loaded on first use
        ctx.distances(o, h, N, 2)  # the next mesh's tree is built ahead
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 1800 * MB, dtype=torch.uint8, device="cuda")
        ctx.set_mesh(X, IEN)
        d, _ = ctx.distances(o, h, N, 0)
        with pytest.raises(_native.SdfGpuError) as e:
            ctx.distances(o, h, N, 2)
        assert "OUT_OF_MEMORY" in str(e.value)
        again, _ = ctx.distances(o, h, N, 0)
        del fill
        torch.cuda.empty_cache()
        u, _ = ctx.distances(o, h, N, 2)
    finally:
        ctx.close()
        torch.cuda.empty_cache()
    fresh = _native.Context(0)
    fresh.set_mesh(X, IEN)
    assert np.array_equal(d, fresh.distances(o, h, N, 0)[0]) and np.array_equal(again, d)
    assert np.array_equal(u, fresh.distances(o, h, N, 2)[0])
    fresh.close()
