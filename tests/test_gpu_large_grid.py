"""The cell sort in a grid of more than 67 million cells (16,384 chunks of its
scan), where the chunk sums become prefix sums in a launch of their own: the
reference numbering against a plain sort, and neighbours and steps against the
same particles in a grid that just holds them."""
import numpy as np
import pytest

from sphera_b200 import Simulation, cases

pytestmark = pytest.mark.gpu

N = 20000


def _box(cells_per_axis):
    c = cases.random_box(n=N, seed=12)
    if cells_per_axis:
        for d in range(3):
            c.params.domain_hi[d] = cells_per_axis * 2.0 * 1.3 * c.params.dx
    return c


def test_more_chunks_than_a_block_adds_up():
    large, small = _box(412), _box(0)
    a, b = Simulation(large), Simulation(small)
    a.upload(large.state)
    b.upload(small.state)
    d = a.diagnostics()
    assert d.n_cells > 16384 * 4096 > b.diagnostics().n_cells
    for _ in range(2):                       # the sums are cleared for the next sort
        cella, icont, order = a.dump_grid()
        count = np.bincount(cella - 1, minlength=d.n_cells)
        assert icont[0] == 1 and np.array_equal(np.diff(icont), count)
        assert np.array_equal(order, np.argsort(cella, kind="stable") + 1)
    ca, la = a.dump_neighbours()
    cb, lb = b.dump_neighbours()
    assert np.array_equal(ca, cb)
    assert all(set(la[i, :ca[i]]) == set(lb[i, :cb[i]]) for i in range(0, N, 7))
    a.step(5)
    b.step(5)
    x, y = a.download().x, b.download().x
    # the sums run in another cell order: rounding of 80 terms, 1e-12 as in the parity tests
    assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)
