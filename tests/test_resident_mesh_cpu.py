"""Which mesh a context computes with, against a stand-in for the library that records the uploads."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from stl2sdf import MeshGrid, SignedDistances, _native


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
    monkeypatch.setitem(_native._default_ctx, 0, ctx)
    return rec, ctx


def test_a_mesh_of_the_same_size_at_a_freed_address_is_a_new_mesh(recorded):
    rec, _ = recorded
    for k in range(50):  # each one usually takes the freed object's address
        mesh = MeshGrid.TriangularMesh(np.eye(3) * (k + 1.0), [[1, 2, 3]])
        SignedDistances._ctx(mesh)
        assert rec.meshes[-1][0, 0] == k + 1.0
        del mesh


def test_changed_arrays_count(recorded):
    rec, _ = recorded
    mesh = MeshGrid.TriangularMesh(np.eye(3), [[1, 2, 3]])
    for scale in (1.0, 2.0, 6.0):
        mesh.X.__imul__(scale / mesh.X[0, 0])
        SignedDistances._ctx(mesh)
        assert rec.meshes[-1][0, 0] == scale


@pytest.mark.parametrize("device", [False, True])
def test_a_refused_mesh_leaves_none_resident(recorded, device):
    rec, ctx = recorded
    X, IEN = np.eye(3), np.array([[1, 2, 3]])
    ctx.set_mesh(X, IEN, key="a")
    ctx.set_mesh(X, IEN, key="a")
    assert len(rec.meshes) == 1
    rec.refuse = True
    with pytest.raises(_native.SdfGpuError):
        if device:
            ctx.set_mesh_device(0, 3, 0, 1)
        else:
            ctx.set_mesh(2.0 * X, IEN, key="b")
    rec.refuse = False
    ctx.set_mesh(X, IEN, key="a")
    assert len(rec.meshes) == 2  # uploaded again
