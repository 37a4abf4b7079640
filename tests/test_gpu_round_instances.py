"""The two register budgets of the float RF / time-dependent kernel give the
same bits in every form that has both: ions of a launch of 22 or 24 warps per
SM (two rounds of 20 warps, one of 24) equal the same ions advanced in slices
below one round, which take the other instance; and of 48 per SM (3 rounds
against 2), where some forms change instance and some do not."""
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

FORMS = {  # precision, integrator, collision, B field, waveform
    "boris": (capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_HSS, False, False),
    "boris-none": (capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_NONE, False, False),
    "boris-B": (capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_LANGEVIN, True, False),
    "boris-wave": (capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_HSS, False, True),
    "rk4": (capi.PREC_MIXED, capi.INTEGRATOR_RK4, capi.COLLISION_HSS, False, False),
    "rk4-none-B": (capi.PREC_MIXED, capi.INTEGRATOR_RK4, capi.COLLISION_NONE, True, False),
    "rk4-wave": (capi.PREC_MIXED, capi.INTEGRATOR_RK4, capi.COLLISION_HSS, False, True),
    "hilo": (capi.PREC_MIXED_HILO, capi.INTEGRATOR_BORIS, capi.COLLISION_HSS, False, False),
    "hilo-none-wave": (capi.PREC_MIXED_HILO, capi.INTEGRATOR_BORIS, capi.COLLISION_NONE, False, True),
}


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


@pytest.mark.parametrize("per_sm", [22, 24, 48])
@pytest.mark.parametrize("form", list(FORMS))
def test_instances_agree_in_every_form(form, per_sm):
    precision, integrator, collision, mag, wave = FORMS[form]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 32 * per_sm * sms
    st = generate_ions(3, [cfg.species_spec(n, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                            {"type": "thermal", "temperature_K": 300.0})])
    ens = _ensembles("trap")
    if mag:
        ens[0].update(magnetic_enabled=1, B_T=[0.0, 0.0, 0.5])
    w = capi.Waveform()                     # linear, 2 V to 1 V in 1 ms
    w.type, w.clamp, w.p[0], w.p[1], w.p[3] = 1, 1, 2.0, 1.0, 1e-3

    def run(s, first):
        with Simulation(ens, precision=precision, integrator=integrator, collision=collision, rng_seed=9) as sim:
            if wave:
                sim.set_waveform(0, 0, w)
            sim.upload(s, first_id=first)
            sim.advance(60)
            return sim.download()

    whole = run(st, 0)
    for lo in (0, (n // 2) // 128 * 128):
        part = run(subset(st, lo, min(lo + 12800, n)), lo)
        for k in ("x", "y", "z", "vx", "vy", "vz", "active"):
            np.testing.assert_array_equal(getattr(whole, k)[lo:lo + 12800], getattr(part, k), err_msg=k)
