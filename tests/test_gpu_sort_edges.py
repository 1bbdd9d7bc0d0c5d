"""The cell sort at the edges of its scan: grids whose cells (with the
removal bin) end just before, on and just after a chunk of 4096, particle
counts around a tile of 256, with and without particles to remove (their
replay shares a launch with the scan).  Whole numbers, equal to the
oracle's."""
import numpy as np
import pytest

from sphera_b200 import Simulation, abi, cases

pytestmark = pytest.mark.gpu


def _case(cells, n, outside):
    """n particles in a grid of cells[0] x cells[1] x cells[2]."""
    c = cases.random_box(n=n, seed=n)
    h2 = 2.0 * c.params.dx * c.params.trunc
    hi = tuple((k - 2) * h2 for k in cells)   # CreaGrid adds 2h on each side
    x = c.state.x / c.meta["side"] * np.array(hi)
    if outside:
        x[:: max(1, n // 5), 2] = hi[2] + 9.0
    prm = c.params
    for d in range(3):
        prm.domain_hi[d] = hi[d]
    st = abi.State(x, c.state.v, c.state.rho, c.state.p, c.state.m)
    return cases.Case(c.name, prm, c.geometry, st)


@pytest.mark.parametrize("outside", [False, True])
@pytest.mark.parametrize("cells,n", [((13, 15, 21), 257), ((16, 16, 16), 256), ((17, 15, 16), 255),
                                     ((4, 3, 3), 1), ((64, 32, 8), 4097)])
def test_grid_at_scan_edges(cells, n, outside, oracle_lib):
    case = _case(cells, n, outside)
    sim = Simulation(case)
    sim.upload(case.state)
    o = oracle_lib.Oracle(case)
    o.prepare()
    assert tuple(sim.diagnostics().grid_ncd) == cells
    if outside and n == 1:
        assert sim.download().n == o.n == 0
        return
    for step in range(2):
        got, want = sim.dump_grid(), o.grid()
        sim.n = o.n
        for a, b in zip(got, want):
            assert np.array_equal(a[:len(b)], b)
        sim.step(1)
        o.step(1)
