"""The planned FP64 step loop (launches of 8 steps or more, uniform field)
against the loop with per-step bookkeeping (launches of up to 7 steps): the
same bits, death and arrival times included, where the plan's rules change:
launches of 8, 9 and many steps, ions that meet a wall or the detector plane
within a few steps, ions outside at the start, a field that is zero, and every
collision kind the loop serves."""
from __future__ import annotations

import numpy as np
import pytest

from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200.sim import Simulation, device_count, generate_ions

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _run(per_launch, steps, td, collision, n=300, mix=False):
    env = {"temperature_K": 300.0, "pressure_Pa": 1000.0, "gas_species": "N2"}
    if mix:
        env["gas_mixture"] = [{"species": "N2", "mole_fraction": 0.7}, {"species": "He", "mole_fraction": 0.3}]
    # a 1.2 mm cylinder around a 0.5 mm cloud: a few ions start outside and
    # many leave or cross the plane at 0.2 mm during the run
    dom = {"instrument": "IMS", "geometry": {"origin_m": [0.0, 0.0, -0.0006], "length_m": 0.0012, "radius_m": 0.0007},
           "env": env, "fields": {"DC": {"EN_Td": td}}}
    ens = cfg.ensemble_params(dom, 150e-20, 4e-9, detector_z_m=2e-4)
    st = generate_ions(21, [cfg.species_spec(n, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                             {"type": "gaussian", "center": [0, 0, 0], "std": [3e-4] * 3},
                                             {"type": "thermal", "temperature_K": 300.0})])
    with Simulation([ens], precision=capi.PREC_FP64, collision=collision, rng_seed=5, steps_per_launch=per_launch) as sim:
        sim.upload(st)
        rs = sim.advance(steps)
        return sim.download(), rs


@pytest.mark.parametrize("collision,mix", [(capi.COLLISION_NONE, False), (capi.COLLISION_HSS, False),
                                           (capi.COLLISION_HSS, True), (capi.COLLISION_LANGEVIN, False)])
@pytest.mark.parametrize("per_launch,steps", [(8, 96), (9, 99), (1000, 400)])
@pytest.mark.parametrize("td", [0.0, 60.0])
def test_planned_steps_equal_single_steps(per_launch, steps, td, collision, mix):
    a, ra = _run(per_launch, steps, td, collision, mix=mix)
    b, rb = _run(7, steps, td, collision, mix=mix)
    for k in ("x", "y", "z", "vx", "vy", "vz", "active", "t_death", "t_arrival"):
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=k)
    for k in ("candidates", "collisions", "rate_overflows", "deaths", "arrivals"):
        assert ra[k] == rb[k], k
    assert ra["deaths"] > 0 and ra["arrivals"] > 0
