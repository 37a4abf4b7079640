"""The default launch shape of an FP64 uniform-field handle is the planned
loop's also after a waveform was set and cleared again: the same bits in the
same time (the shape with 10 pending lanes and 8 steps a vote takes 1.14 times
as long here; the bound allows 6 %)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import config0_ensemble, config0_ions
from icarion_b200 import _capi as capi
from icarion_b200.sim import Simulation, device_count

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def test_shape_comes_back_when_the_waveform_is_cleared():
    st = config0_ions(262_144)
    w = capi.Waveform()                       # constant 0 V
    ms, outs = {}, {}
    for cleared in (False, True):
        with Simulation([config0_ensemble()], precision=capi.PREC_FP64, collision=capi.COLLISION_HSS,
                        rng_seed=5) as sim:
            if cleared:
                sim.set_waveform(0, 0, w)
                sim.set_waveform(0, 0, None)
            sim.upload(st)
            ms[cleared] = min(sim.advance(1000)["device_ms"] for _ in range(6))
            outs[cleared] = sim.download()
    for k in ("x", "y", "z", "vx", "vy", "vz", "active"):
        np.testing.assert_array_equal(getattr(outs[False], k), getattr(outs[True], k))
    assert ms[True] <= 1.06 * ms[False], ms
