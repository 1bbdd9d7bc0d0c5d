"""The pair passes with four lanes to a particle and with one: rates of a step
against the oracle where the passes change over (an SM's share of warps) and
where lists are shorter than a lane's share (no neighbour, one, a chunk less
or more one).  FP64 within 1e-12 and nearly all values equal; FP32c within
1e-5 (the bars of the rates on an identical state)."""
import numpy as np
import pytest

from sphera_b200 import Simulation, abi, cases

pytestmark = pytest.mark.gpu


def _sparse(precision):
    """Lists of 0 to about 12 entries, most shorter than a chunk."""
    c = cases.random_box(n=900, seed=7, precision=precision)
    L = 0.35
    for d in range(3):
        c.params.domain_hi[d] = L
    x = c.state.x / c.meta["side"] * L
    return cases.Case(c.name, c.params, c.geometry, abi.State(x, c.state.v, c.state.rho, c.state.p, c.state.m))


# tiles of 256 particles against 7, 5 and 8 warps on each of 148 SMs
CASES = {
    "sparse": _sparse,
    "one_tile": lambda p: cases.random_box(n=256, seed=8, precision=p),
    "box_33024": lambda p: cases.random_box(n=129 * 256, seed=9, precision=p),
    "box_33025": lambda p: cases.random_box(n=129 * 256 + 1, seed=9, precision=p),
    "box_23552": lambda p: cases.random_box(n=92 * 256, seed=10, precision=p),
    "box_23553": lambda p: cases.random_box(n=92 * 256 + 1, seed=10, precision=p),
    "box_37633": lambda p: cases.random_box(n=147 * 256 + 1, seed=11, precision=p),
    "corner_2d": lambda p: cases.dam_break_2d(dx=0.04, tank=(0.4, 0.4), column=(0.4, 0.4), jitter=0.2, precision=p),
}


@pytest.mark.parametrize("precision", [abi.SPH_PREC_FP64, abi.SPH_PREC_FP32C])
@pytest.mark.parametrize("name", list(CASES))
def test_rates_and_a_step(name, precision, oracle_lib):
    case = CASES[name](precision)
    sim = Simulation(case)
    sim.upload(case.state)
    o = oracle_lib.Oracle(case)
    o.prepare()
    acc, dden = sim.rhs_momentum(), sim.continuity()
    o.rhs_momentum()
    o.continuity()
    s = o.get()
    tol = 1e-12 if precision == abi.SPH_PREC_FP64 else 1e-5
    for got, want in ((acc, s["acc"]), (dden, s["dden"])):
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
        if precision == abi.SPH_PREC_FP64:
            assert np.mean(got == want) > 0.99
    step, two = Simulation(case), oracle_lib.Oracle(case)
    step.upload(case.state)
    two.prepare()
    step.step(2)
    two.step(2)
    x = two.get()["x"]
    assert np.linalg.norm(step.download().x - x) <= (1e-12 if precision == abi.SPH_PREC_FP64 else 1e-8) * np.linalg.norm(x)
