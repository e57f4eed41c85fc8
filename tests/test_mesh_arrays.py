"""Meshes as arrays: mesh_to_numpy copies and leaves the mesh, whoever owns its memory;
take_mesh hands the library's buffer over."""
import ctypes
import gc

import numpy as np

from libfluid_gb300 import capi


def _triangles(n):
    return np.arange(21 * n, dtype=np.float32).reshape(n, 21)


def test_a_copy_leaves_the_mesh_to_its_owner():
    own = _triangles(5)
    mesh = capi.Mesh()
    mesh.triangles, mesh.n, mesh.capacity = own.ctypes.data_as(capi.P(capi.MeshTriangle)), 5, 5
    first = capi.mesh_to_numpy(mesh)
    first[:] = 0
    second = capi.mesh_to_numpy(mesh)
    assert (second == _triangles(5)).all() and (own == second).all()
    assert mesh.n == 5 and mesh.capacity == 5 and ctypes.addressof(mesh.triangles.contents) == own.ctypes.data
    del first, second
    gc.collect()
    assert (own == _triangles(5)).all()


def test_a_taken_mesh_lives_as_long_as_its_views():
    libc = ctypes.CDLL(None)
    libc.malloc.restype, libc.malloc.argtypes = ctypes.c_void_p, [ctypes.c_size_t]
    at = libc.malloc(8 * ctypes.sizeof(capi.MeshTriangle))
    want = _triangles(5)
    ctypes.memmove(at, want.ctypes.data, want.nbytes)
    mesh = capi.Mesh()
    mesh.triangles, mesh.n, mesh.capacity = ctypes.cast(at, capi.P(capi.MeshTriangle)), 5, 8
    taken = capi.take_mesh(mesh)
    assert not mesh.triangles and mesh.n == 0 and mesh.capacity == 0
    capi.load().fgb_mesh_free(ctypes.byref(mesh))  # nothing left to free
    assert taken.ctypes.data == at
    view = taken[2:, :9]
    del taken
    gc.collect()
    assert (view == want[2:, :9]).all()
    assert len(capi.take_mesh(capi.Mesh())) == 0 and len(capi.mesh_to_numpy(capi.Mesh())) == 0
