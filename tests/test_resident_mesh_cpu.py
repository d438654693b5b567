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

    def sdfgpu_set_mesh(self, ctx, X, nnp, IEN, nel):
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
