"""Which mesh a context takes for its resident one (Context.set_mesh with a TriangularMesh's key), against a
stand-in for the library that records the uploads."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from stl2sdf import MeshGrid, _native


class Recorder:
    def __init__(self):
        self.meshes = []
        self.refuse = False

    def sdfgpu_set_mesh_device(self, ctx, X, nnp, IEN, nel):
        return 1

    def sdfgpu_set_mesh(self, ctx, X, nnp, IEN, nel):
        if self.refuse:
            return 1
        self.meshes.append(np.ctypeslib.as_array(ctypes.cast(X, ctypes.POINTER(ctypes.c_double)), (nnp, 3)).copy())
        return 0

    def sdfgpu_last_error(self, ctx):
        return b"refused"


@pytest.fixture
def recorded(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(_native, "lib", lambda: rec)
    ctx = _native.Context.__new__(_native.Context)
    ctx._p, ctx._mesh_key = None, None
    return rec, ctx


IEN = np.array([[1, 2, 3]])


def test_a_mesh_of_the_same_size_at_a_freed_address_is_a_new_mesh(recorded):
    rec, ctx = recorded
    for k in range(50):  # each one usually takes the freed object's address
        mesh = MeshGrid.TriangularMesh(np.eye(3) * (k + 1.0), IEN)
        for _ in range(2):  # the second call finds it resident
            ctx.set_mesh(mesh.vertex_rows(), mesh.triangle_rows(), key=mesh._key)
        del mesh
    assert [m[0, 0] for m in rec.meshes] == [k + 1.0 for k in range(50)]


@pytest.mark.parametrize("device", [False, True])
def test_a_refused_mesh_leaves_none_resident(recorded, device):
    rec, ctx = recorded
    mesh, bad = (MeshGrid.TriangularMesh(np.eye(3) * s, IEN) for s in (1.0, 2.0))
    ctx.set_mesh(mesh.vertex_rows(), mesh.triangle_rows(), key=mesh._key)
    rec.refuse = True
    with pytest.raises(_native.SdfGpuError):
        if device:
            ctx.set_mesh_device(0, 3, 0, 1)
        else:
            ctx.set_mesh(bad.vertex_rows(), bad.triangle_rows(), key=bad._key)
    rec.refuse = False
    ctx.set_mesh(mesh.vertex_rows(), mesh.triangle_rows(), key=mesh._key)
    assert len(rec.meshes) == 2  # uploaded again
