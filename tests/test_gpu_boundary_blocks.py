"""The 2D wall integrals in blocks of 128 threads (from 8 tiles of 256 particles
an SM in the FP32c form) and of 256 (the FP64 form at the same size): both are
FP64 passes over the same positions, so their entries are equal bit for bit, and
close sides equal the oracle's.  A full tank: its four corners lie in four places
of the order, and a last tile that is not full."""
import numpy as np
import pytest
import torch

from sphera_b200 import Batch, Simulation, abi, cases

pytestmark = pytest.mark.gpu


def _tank(precision):
    return cases.dam_break_2d(dx=0.0024, tank=(1.0, 2.0), column=(1.0, 2.0), jitter=0.2, precision=precision)


def test_both_block_sizes_give_the_same_entries(oracle_lib):
    case = _tank(abi.SPH_PREC_FP32C)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = (case.n + 255) // 256
    assert 8 * sms <= tiles < 32 * sms and case.n % 256
    got = []
    for c in (case, _tank(abi.SPH_PREC_FP64)):
        sim = Simulation(c)
        sim.upload(c.state)
        got.append(sim.dump_boundary(4))
        sim.close()
    n, clob, vals = got[0]
    assert (n == 2).sum() >= 16
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    o = oracle_lib.Oracle(case)
    o.prepare()
    on, oc, ov = o.boundary(4)
    assert np.array_equal(n, on) and np.array_equal(clob, oc)
    near = n > 0
    assert np.linalg.norm(vals[near] - ov[near]) <= 1.0e-12 * np.linalg.norm(ov[near])


@pytest.mark.parametrize("precision", [abi.SPH_PREC_FP64, abi.SPH_PREC_FP32C])
def test_members_of_a_3d_batch_have_their_own_entries(precision):
    """The 3D integrals number the chunks of 128 members at a time: members on
    both sides of that, of unequal sizes, one without particles near a wall's
    end and one without any, each bit for bit as alone."""
    cs = [cases.dam_break_3d(dx=0.06 if i % 3 else 0.05, jitter=0.1, seed=i, precision=precision) for i in range(131)]
    empty = cs[126]
    none = abi.State.empty(0)
    batch = Batch(cs)
    states = [c.state for c in cs]
    states[126] = none
    batch.upload(states)
    batch.step(6)
    for i in (0, 1, 3, 125, 127, 128, 130):
        alone = Simulation(cs[i])
        alone.upload(cs[i].state)
        alone.step(6)
        a, b = alone.download(), batch.download(i)
        for f in ("x", "v", "rho", "p"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), (i, f)
        alone.close()
    assert batch.download(126).n == 0 and empty.n > 0
