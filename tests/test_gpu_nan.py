"""A particle whose position has become NaN between the calls of a host's own
time loop is not passed over by the pair sums of the FP64 form: whatever is
summed over it is NaN too, so the host sees the fault where it arises."""
import numpy as np
import pytest

from sphera_b200 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_a_nan_separation_reaches_every_sum_over_it(dim):
    case = cases.dam_break_2d(dx=0.08, jitter=0.1) if dim == 2 else cases.dam_break_3d(dx=0.05, jitter=0.1)
    case.params.teta_p = 0.2
    i = case.n // 2
    case.state.v[i, 0] = np.nan
    sim = Simulation(case)
    sim.upload(case.state)
    counts, lists = sim.dump_neighbours(sim.diagnostics().nmaxpartj)
    touched = {i} | {q for q in range(case.n) if i + 1 in lists[q, :counts[q]]}
    assert len(touched) > 5
    sim.leapfrog_trajectories()          # its position is NaN, the lists are not
    acc, dden = sim.rhs_momentum(), sim.continuity()
    sim.eos()                            # with the partial smoothing of the pressures
    st = sim.download()
    assert set(np.flatnonzero(np.isnan(st.x).any(axis=1))) == {i}
    assert set(np.flatnonzero(np.isnan(acc).any(axis=1))) == touched
    assert set(np.flatnonzero(np.isnan(dden))) == touched
    assert set(np.flatnonzero(np.isnan(st.p))) == touched
    assert set(np.flatnonzero(np.isnan(st.rho))) == touched
