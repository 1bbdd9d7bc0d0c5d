"""The neighbour search where its scan branches: groups of few particles and
whole warps, blocks of few candidates and of many tiles, lists far longer than
a lane's waiting entries, lists at NMAXPARTJ, thin columns (a warp over many z
cells), coordinates far from the origin, and simulations on both sides of the
change in what a particle taken singly is held to cost.  Whole numbers: counts and lists equal to the oracle's, in its
order."""
import numpy as np
import pytest

from sphera_b200 import Simulation, abi, cases

pytestmark = pytest.mark.gpu


def _box(x, coef=None, shift=0.0):
    c = cases.random_box(n=len(x), seed=3)
    prm = c.params
    for d in range(3):
        prm.domain_lo[d] = shift
        prm.domain_hi[d] = shift + 0.35
    if coef:
        prm.coef_nmaxpartj = coef
    st = abi.State(x + shift, c.state.v, c.state.rho, c.state.p, c.state.m)
    return cases.Case(c.name, prm, c.geometry, st)


def _uniform(n, side, seed=1):
    return np.random.default_rng(seed).uniform(0.0, side, size=(n, 3))


def _clusters(sizes, radius=0.008, seed=2):
    rng = np.random.default_rng(seed)
    x = []
    for k in sizes:
        centre = rng.uniform(0.02, 0.33, size=3)
        x.append(centre + rng.uniform(-radius, radius, size=(k, 3)))
    return np.concatenate(x)


def _columns(seed=4):
    rng = np.random.default_rng(seed)
    z = np.linspace(0.001, 0.349, 60)
    x = [np.column_stack([np.full(60, a) + rng.uniform(-1e-3, 1e-3, 60), np.full(60, b), z])
         for a in (0.05, 0.08, 0.2) for b in (0.05, 0.1, 0.3)]
    return np.concatenate(x)


CASES = {
    "one": (lambda: np.array([[0.1, 0.1, 0.1]]), None, 0.0),
    "sparse": (lambda: _uniform(500, 0.35), None, 0.0),
    "ordinary": (lambda: _uniform(4000, 0.16), None, 0.0),
    "crowded": (lambda: _uniform(4000, 0.12), 3.0, 0.0),
    "cells_of_15_to_33": (lambda: _clusters([15, 16, 17, 31, 32, 33, 1, 2], radius=0.004), None, 0.0),
    "long_lists": (lambda: _clusters([100, 115, 116, 117, 118, 140, 200]), 3.0, 0.0),
    "at_the_cap": (lambda: _clusters([41, 42, 43, 44, 45, 60, 130]), 0.3, 0.0),
    "at_the_cap_dense": (lambda: _uniform(4000, 0.12), 0.3, 0.0),
    "thin_columns": (_columns, None, 0.0),
    "far_from_origin": (lambda: _uniform(4000, 0.16), None, 1000.0),
}


# from 296 tiles of 256 particles on (two to each of 148 SMs) a particle taken
# singly weighs less against its group's common window: columns about a warp's
# particles apart, both cell widths, 2D
LARGE = {
    "dam_94221": lambda: cases.dam_break_3d(dx=0.0105, jitter=0.1, seed=5),
    "box_75777": lambda: cases.random_box(n=296 * 256 + 1, seed=5),
    "column_2d_80000": lambda: cases.dam_break_2d(dx=0.005, jitter=0.1, seed=5),
}


@pytest.mark.parametrize("name", list(CASES) + list(LARGE))
def test_lists_equal_oracle(name, oracle_lib):
    if name in LARGE:
        case = LARGE[name]()
    else:
        make, coef, shift = CASES[name]
        case = _box(make(), coef, shift)
    sim = Simulation(case)
    sim.upload(case.state)
    o = oracle_lib.Oracle(case)
    o.prepare()
    nm = o.nmaxpartj
    gc, gl = sim.dump_neighbours(nm)
    oc, ol = o.neighbours(nm)
    assert np.array_equal(gc, oc)
    assert np.array_equal(gl, ol)
    warned = bool(sim.diagnostics().warnings & abi.SPH_WARN_NEIGHBOURS_TRUNCATED)
    assert warned == (o.truncated > 0)
