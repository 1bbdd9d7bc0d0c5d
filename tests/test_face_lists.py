"""The face lists of the cells (host, on creation) take time in proportion to
the faces that they hold: a wall of strips that all cross the same cells beside
a wall of as many small faces.  Without a device: sph_memory_required prepares
the simulation as sph_create does."""
import ctypes as C
import time

import numpy as np

import sphera_b200
from sphera_b200 import abi, cases

L = 0.4


def _floor(nx, ny, width):
    """A floor of nx x ny faces, `width` of its L in y."""
    xs, ys = np.linspace(0.0, L, nx + 1), np.linspace(0.0, width, ny + 1)
    V = np.array([[x, y, 0.0] for y in ys for x in xs])

    def at(i, j):
        return j * (nx + 1) + i + 1

    F = [[at(i, j), at(i + 1, j), at(i + 1, j + 1), at(i, j + 1)] for j in range(ny) for i in range(nx)]
    return abi.Geometry(V, [abi.make_zone()], faces=F, face_zone=np.ones(len(F), dtype=np.int32))


def _seconds(geometry):
    p = cases._params(3, 0.01, (0.0, 0.0, 0.0), (L, L, L))
    p.max_close_bound_faces = 10000
    cap, out = np.array([1000], np.int32), C.c_uint64()
    t = []
    for _ in range(3):
        t0 = time.perf_counter()
        rc = sphera_b200.lib().sph_memory_required(1, C.byref(p), C.byref(geometry.struct), abi.iptr(cap), C.byref(out))
        t.append(time.perf_counter() - t0)
        assert rc == abi.SPH_OK
    return min(t)


def test_time_is_linear_in_the_faces_of_a_cell():
    strips = _seconds(_floor(1, 3600, 0.02))     # every cell of a row holds all of them
    spread = _seconds(_floor(60, 60, L))         # a cell holds about 25
    assert strips < 2.0 * spread + 0.05, (strips, spread)
