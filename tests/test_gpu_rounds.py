"""The float RF / time-dependent kernel has two register budgets, chosen by
the launch's rounds of resident warps.  Around the sizes where the choice
changes (20 and 24 warps of 32 ions per SM) the two instances give the same
bits: ions of a large launch equal the same ions advanced in a launch of
their own block-aligned slice."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200.sim import Simulation, device_count, generate_ions
from icarion_b200.sweep import subset
from test_gpu_rf_table import _ensembles

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


@pytest.mark.parametrize("extra", [1, 33, 4000])
@pytest.mark.parametrize("per_sm", [20, 24])
def test_instances_agree(per_sm, extra):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 32 * per_sm * sms + extra
    st = generate_ions(3, [cfg.species_spec(n, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                            {"type": "thermal", "temperature_K": 300.0})])
    ens = _ensembles("trap")

    def run(s, first):
        with Simulation(ens, precision=capi.PREC_MIXED, collision=capi.COLLISION_HSS, rng_seed=9) as sim:
            sim.upload(s, first_id=first)
            sim.advance(60)
            return sim.download()

    whole = run(st, 0)
    for lo in (0, (n // 2) // 128 * 128):
        part = run(subset(st, lo, min(lo + 12800, n)), lo)
        for k in ("x", "y", "z", "vx", "vy", "vz", "active"):
            np.testing.assert_array_equal(getattr(whole, k)[lo:lo + 12800], getattr(part, k))
