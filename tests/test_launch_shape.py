"""A launch configuration that names some of its entries leaves the others at
their defaults: 0 blocks, and -1 for a pair loop, whose 0 is the lean loop."""
import ctypes as C

import pytest

import sphera_b200
from sphera_b200 import SphError, Simulation, abi, cases


class _Recorder:
    def sph_set_launch_shape(self, h, shape):
        self.shape = [shape[i] for i in range(7)]
        return abi.SPH_OK


@pytest.mark.parametrize("given, want", [
    ({}, [0, 0, 0, 0, 0, -1, -1]),
    ({"lists": 296}, [296, 0, 0, 0, 0, -1, -1]),
    ({"momentum_shape": 0}, [0, 0, 0, 0, 0, 0, -1]),
    ({"continuity": 148, "continuity_shape": 2}, [0, 0, 148, 0, 0, -1, 2]),
])
def test_missing_entries_are_the_defaults(monkeypatch, given, want):
    lib = _Recorder()
    monkeypatch.setattr(sphera_b200, "lib", lambda: lib)
    sphera_b200._set_launch_shape(C.c_void_p(), given)
    assert lib.shape == want


@pytest.mark.gpu
def test_shapes_outside_the_loops_are_refused():
    case = cases.dam_break_2d(dx=0.04)
    sim = Simulation(case)
    sim.upload(case.state)
    for ok in ({}, {"momentum_shape": -1, "continuity_shape": -1}, {"momentum_shape": 2, "continuity_shape": 2}):
        sim.set_launch_shape(ok)
    for bad in ({"momentum_shape": -2}, {"continuity_shape": 3}, {"lists": -1}):
        with pytest.raises(SphError) as e:
            sim.set_launch_shape(bad)
        assert e.value.code == abi.SPH_ERR_INVALID_ARGUMENT
