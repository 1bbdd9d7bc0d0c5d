"""The pair passes with one lane to a particle, which simulations of 38,000
particles and more run (smaller ones without C1 take four lanes, the FP32c form
up to 19,000 in the momentum pass, whatever their launch shape): each loop shape against the oracle beside walls, all shapes and
grids against one another bit for bit, and a member's results with four lanes,
alone, against those with one, in a batch that fills the SMs."""
import numpy as np
import pytest
import torch

from sphera_b200 import Batch, Simulation, abi, cases

pytestmark = pytest.mark.gpu

FORMS = [abi.SPH_PREC_FP64, abi.SPH_PREC_FP32C]

SHAPES = [dict(momentum_shape=0, continuity_shape=0),
          dict(momentum_shape=1, continuity_shape=1),
          dict(momentum_shape=2, continuity_shape=2),
          dict(momentum_shape=1, continuity_shape=0, lists=148, momentum=40, continuity=100, boundary=60),
          {}]


def _moving(case):
    """A column in collapse: it spreads along x as it falls."""
    st = case.state
    lx, lz = st.x[:, 0].max(), st.x[:, 2].max()
    st.v[:, 0] = 0.8 * st.x[:, 0] / lx
    st.v[:, 2] = -0.8 * (lz / lx) * st.x[:, 2] / lz
    st.v[:, 0 if case.params.dim == 2 else 1] += 0.02 * np.sin(40.0 * st.x[:, 2])
    return case


def _case(dim, precision):
    c = cases.dam_break_2d(dx=0.0069, jitter=0.1, precision=precision) if dim == 2 else \
        cases.dam_break_3d(dx=0.0135, jitter=0.1, precision=precision)
    # eight warps an SM and more: one lane in all pair passes
    assert (c.n + 255) // 256 >= torch.cuda.get_device_properties(0).multi_processor_count
    return _moving(c)


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("dim", [2, 3])
def test_every_shape_on_the_oracle_and_the_same_bits(dim, precision, oracle_lib):
    case = _case(dim, precision)
    o = oracle_lib.Oracle(case)
    o.prepare()
    o.rhs_momentum()
    o.continuity()
    want = o.get()
    tol = 1e-12 if precision == abi.SPH_PREC_FP64 else 1e-5   # the bars of the rates on an identical state
    first = None
    for shape in SHAPES:
        sim = Simulation(case)
        sim.upload(case.state)
        sim.set_launch_shape(shape)
        acc, dden = sim.rhs_momentum(), sim.continuity()
        assert np.linalg.norm(acc - want["acc"]) <= tol * np.linalg.norm(want["acc"]), shape
        assert np.linalg.norm(dden - want["dden"]) <= tol * np.linalg.norm(want["dden"]), shape
        sim.upload(case.state)
        sim.step(8)
        st = sim.download()
        sim.close()
        got = (acc, dden, st.x, st.v, st.rho, st.p)
        if first is None:
            first = got
        assert all(np.array_equal(a, b) for a, b in zip(got, first)), shape


# either side of four warps an SM (FP32c momentum) and, in 2D, of six (FP32c
# continuity) on 148 SMs: 73 and 74 tiles of 256 particles, 110 and 111
EDGES = {
    "box_73": lambda: cases.random_box(n=73 * 256, seed=21, precision=abi.SPH_PREC_FP32C),
    "box_74": lambda: cases.random_box(n=74 * 256, seed=21, precision=abi.SPH_PREC_FP32C),
    "column_110": lambda: _moving(cases.dam_break_2d(dx=0.00845, jitter=0.1, precision=abi.SPH_PREC_FP32C)),
    "column_111": lambda: _moving(cases.dam_break_2d(dx=0.0084, jitter=0.1, precision=abi.SPH_PREC_FP32C)),
}


@pytest.mark.parametrize("name", list(EDGES))
def test_fp32c_rates_where_lanes_change_over(name, oracle_lib):
    case = EDGES[name]()
    assert (case.n + 255) // 256 == int(name.split("_")[1])
    o = oracle_lib.Oracle(case)
    o.prepare()
    o.rhs_momentum()
    o.continuity()
    want = o.get()
    sim = Simulation(case)
    sim.upload(case.state)
    for got, ref in ((sim.rhs_momentum(), want["acc"]), (sim.continuity(), want["dden"])):
        assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("precision", FORMS)
@pytest.mark.parametrize("dim", [2, 3])
def test_four_lanes_alone_equal_one_lane_in_a_batch(dim, precision):
    small = _moving(cases.dam_break_2d(dx=0.03, jitter=0.1, precision=precision) if dim == 2 else
                    cases.dam_break_3d(dx=0.03, jitter=0.1, precision=precision))
    alone = Simulation(small)
    alone.upload(small.state)
    alone.step(12)
    a = alone.download()
    batch = Batch([small, _case(dim, precision)])
    batch.upload()
    batch.step(12)
    b = batch.download(0)
    for f in ("x", "v", "rho", "p"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
