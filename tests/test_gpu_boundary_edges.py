"""The wall integrals where their passes branch: 2D corner particles (two
close sides; a tank so small that all four corners share a block), 3D
faces that the projected hemisphere overlaps the edges of, faces it lies
inside, and triangles.  Close faces equal to the oracle's, integrals within
1e-12 (the bar of the boundary data)."""
import numpy as np
import pytest

from sphera_b200 import Simulation, abi, cases

pytestmark = pytest.mark.gpu

TOL = 1.0e-12


def _corners():
    return cases.dam_break_2d(dx=0.04, tank=(0.4, 0.4), column=(0.4, 0.4), jitter=0.2)


def _small_box():
    return cases.dam_break_3d(dx=0.02, tank=(0.1, 0.12, 0.1), block=(0.1, 0.12, 0.1), jitter=0.2)


def _large_box():
    return cases.dam_break_3d(dx=0.04, tank=(0.8, 0.6, 0.6), block=(0.8, 0.6, 0.6), jitter=0.2)


def _triangles():
    c = _large_box()
    F = c.geometry.faces
    tri = np.concatenate([np.column_stack([F[:, 0], F[:, 1], F[:, 2], 0 * F[:, 0]]),
                          np.column_stack([F[:, 0], F[:, 2], F[:, 3], 0 * F[:, 0]])]).astype(np.int32)
    g = abi.Geometry(c.geometry.vertices, c.geometry.zones, faces=tri, face_zone=np.ones(len(tri), np.int32))
    return cases.Case(c.name, c.params, g, c.state)


@pytest.mark.parametrize("make", [_corners, _small_box, _large_box, _triangles])
def test_boundary_entries(make, oracle_lib):
    case = make()
    case.params.bdt_capacity = 8 * case.n
    sim = Simulation(case)
    sim.upload(case.state)
    o = oracle_lib.Oracle(case)
    o.prepare()
    gn, gc, gv = sim.dump_boundary(8)
    on, oc, ov = o.boundary(8)
    assert np.array_equal(gn, on) and np.array_equal(gc, oc)
    assert (gn > 1).sum() >= 8
    near = gn > 0
    assert np.linalg.norm(gv[near] - ov[near]) <= TOL * np.linalg.norm(ov[near])
