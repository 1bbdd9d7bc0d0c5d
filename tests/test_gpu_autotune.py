"""What the tuner chooses from: 1 to 32 blocks an SM below one block to a tile of
256 particles, and one block to a tile; nothing for pair passes that run four
lanes to a particle.  A tuned simulation steps bit for bit as an untuned one."""
import numpy as np
import pytest
import torch

from sphera_b200 import Simulation, abi, cases

pytestmark = pytest.mark.gpu

TILE_CLASSES = ("lists", "momentum", "continuity", "boundary")

# 53 tiles: four lanes to a particle in every pair pass; 497: one lane; 4,928:
# more tiles than 32 blocks on each of 148 SMs
CASES = {
    "dam_13500": (lambda p: cases.dam_break_3d(dx=0.02, jitter=0.1, precision=p), 12),
    "dam_127008": (lambda p: cases.dam_break_3d(dx=0.0095, jitter=0.1, precision=p), 5),
    "column_1261378": (lambda p: cases.dam_break_2d(dx=0.00126, jitter=0.1, precision=p), 3),
}


@pytest.mark.parametrize("precision", [abi.SPH_PREC_FP64, abi.SPH_PREC_FP32C])
@pytest.mark.parametrize("name", list(CASES))
def test_choices_and_results(name, precision):
    make, steps = CASES[name]
    case = make(precision)
    tiles = (case.n + 255) // 256
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    allowed = {sms * m for m in (1, 2, 4, 8, 16, 32) if sms * m < tiles} | {tiles}
    tuned, plain = Simulation(case), Simulation(case)
    tuned.upload(case.state)
    plain.upload(case.state)
    got = tuned.autotune(reps=1)
    assert all(got[k] in allowed for k in TILE_CLASSES), got
    if tiles * 8 < 5 * sms:
        assert got["momentum"] == got["continuity"] == tiles
        fp32c = precision == abi.SPH_PREC_FP32C
        assert (got["momentum_shape"], got["continuity_shape"]) == ((2, 2) if fp32c else (0, 1))
    tuned.step(steps)
    plain.step(steps)
    a, b = tuned.download(), plain.download()
    for f in ("x", "v", "rho", "p"):
        assert np.array_equal(getattr(a, f), getattr(b, f))
