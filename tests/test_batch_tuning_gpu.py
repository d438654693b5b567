"""What a batch with autotuning runs besides its items."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_items_without_tiles_are_not_tuned(torus_mesh, mode):
    """The scatter takes this item and has no tiles: tuning them would run the tile fold, whose buffers (the
    (tile, triangle) pairs alone take 13 MB) show in the device's free memory."""
    import torch
    from stl2sdf import _native

    X, IEN = torus_mesh
    o, _, N, h, _ = _native.grid_setup(X.min(0), X.max(0), 121, 3)

    def used(autotune):
        ctx = _native.Context(0)
        before = torch.cuda.mem_get_info()[0]
        field = ctx.sdf_batch([(X, IEN, o, h, N)], mode, streams=1, autotune=autotune)[0]
        taken = before - torch.cuda.mem_get_info()[0]
        ctx.close()
        return taken, field

    torch.cuda.init()
    used(False), used(True)  # kernels are loaded on first use, into device memory
    (plain, a), (tuned, b) = used(False), used(True)
    assert plain > 0 and abs(tuned - plain) < 4 << 20
    assert np.array_equal(a, b)
