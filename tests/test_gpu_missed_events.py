"""Ions whose stored clock event was not taken when its step went by: they
were inactive then (icb_update_state, icb_advance_host), the engine clock was
moved past it (icb_set_clock), or the caller's step left collisions out
(push and finalize without collide).  And ions whose wait for an event began
after the step that the engine clock was moved back to.

The planned FP64 loop (launches of 8 steps or more) and the loop with
per-step bookkeeping (up to 7) give the same bits from such a state on, the
ions go on colliding at the rate they had, and the FP64 run follows the
oracle (the tolerances of the oracle comparisons elsewhere: 1e-9 for 99 % of
the ions, 1 % of the collisions)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from helpers import oracle_state
from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200.sim import Simulation, device_count, generate_ions

pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "vx", "vy", "vz", "active", "t_death", "t_arrival")
COUNTS = ("candidates", "collisions", "rate_overflows", "deaths", "arrivals")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _domain(mix=False):
    # 100 Pa of N2: a candidate event every 14 steps
    env = {"temperature_K": 300.0, "pressure_Pa": 100.0, "gas_species": "N2"}
    if mix:
        env["gas_mixture"] = [{"species": "N2", "mole_fraction": 0.7}, {"species": "He", "mole_fraction": 0.3}]
    dom = {"instrument": "IMS", "geometry": {"origin_m": [0.0, 0.0, -0.02], "length_m": 0.04, "radius_m": 0.02},
           "env": env, "fields": {"DC": {"EN_Td": 20.0}}}
    return cfg.ensemble_params(dom, 150e-20, 4e-9)


def _ions(n=300):
    return generate_ions(21, [cfg.species_spec(n, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                               {"type": "gaussian", "center": [0, 0, 0], "std": [3e-4] * 3},
                                               {"type": "thermal", "temperature_K": 300.0})])


def _miss(sim, how, steps):
    """Lets the events of `steps` steps go by for every second ion, or for all."""
    if how == "rewound":
        sim.set_clock(0, np.zeros(1))
    elif how == "clock":
        step, t = sim.clock()
        sim.set_clock(step + steps, t + steps * 4e-9)
    elif how == "uncollided":
        for _ in range(steps):
            sim.step_batch()
            sim.finalize()
    else:
        idle = sim.download()
        idle.active[::2] = 0
        sim.update_state(idle)
        if how == "host":
            sim.advance_host(idle, steps, n_chunks=2)
        else:
            sim.advance(steps)
            idle = sim.download()
        idle.active[:] = 1
        if how == "update":
            sim.update_state(idle)
        else:
            sim.advance_host(idle, 9, n_chunks=2)


def _run(per_launch, how, missed, precision=capi.PREC_FP64, collision=capi.COLLISION_HSS, mix=False):
    with Simulation([_domain(mix)], precision=precision, collision=collision, rng_seed=5,
                    steps_per_launch=per_launch) as sim:
        sim.upload(_ions())
        sim.advance(30 if how != "rewound" else 300)
        _miss(sim, how, missed)
        rs = sim.advance(200)
        return sim.download(), rs


@pytest.mark.parametrize("collision,mix", [(capi.COLLISION_HSS, False), (capi.COLLISION_HSS, True),
                                           (capi.COLLISION_LANGEVIN, False)])
@pytest.mark.parametrize("missed", [1, 2, 40])
@pytest.mark.parametrize("how", ["update", "host", "clock", "uncollided"])
def test_planned_steps_equal_single_steps_after_missed_events(how, missed, collision, mix):
    b, rb = _run(7, how, missed, collision=collision, mix=mix)
    for per_launch in (8, 1000):
        a, ra = _run(per_launch, how, missed, collision=collision, mix=mix)
        for k in STATE:
            np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=k)
        for k in COUNTS:
            assert ra[k] == rb[k], k


@pytest.mark.parametrize("precision,collision,mix", [(capi.PREC_FP64, capi.COLLISION_HSS, False),
                                                     (capi.PREC_MIXED, capi.COLLISION_HSS, False),
                                                     (capi.PREC_MIXED, capi.COLLISION_HSS, True),
                                                     (capi.PREC_MIXED_HILO, capi.COLLISION_HSS, False),
                                                     (capi.PREC_MIXED, capi.COLLISION_LANGEVIN, False)])
@pytest.mark.parametrize("per_launch", [1, 7, 1000])
@pytest.mark.parametrize("how", ["update", "clock", "rewound", "uncollided"])
def test_collisions_go_on_after_missed_events(how, per_launch, precision, collision, mix):
    """Counts of 200 steps after 40 missed ones against the same 200 steps
    taken at once: both Poisson-like, 5 sigma of their difference apart."""
    _, got = _run(per_launch, how, 40, precision, collision, mix)
    with Simulation([_domain(mix)], precision=precision, collision=collision, rng_seed=6) as sim:
        sim.upload(_ions())
        want = sim.advance(200)
    assert want["collisions"] > 500
    assert abs(got["collisions"] - want["collisions"]) <= 5 * np.sqrt(2 * want["collisions"])


@pytest.mark.parametrize("collision", [capi.COLLISION_HSS, capi.COLLISION_LANGEVIN])
@pytest.mark.parametrize("missed", [1, 40])
@pytest.mark.parametrize("how", ["update", "clock", "rewound"])
def test_fp64_run_after_missed_events_matches_oracle(how, missed, collision):
    out, rs = _run(1000, how, missed, collision=collision)
    ens, ost = _domain(), oracle_state(_ions())
    kind = 2 if collision == capi.COLLISION_HSS else 3
    r = orc.run(ens, ost, 30 if how != "rewound" else 300, collision=kind, seed=5)
    step = 30 + missed if how != "rewound" else 0
    if how == "update":
        ost["active"][::2] = 0
        r = orc.run(ens, ost, missed, collision=kind, seed=5, step0=30, t0=30 * 4e-9, clock=r["clock"])
        ost["active"][:] = 1
    r = orc.run(ens, ost, 200, collision=kind, seed=5, step0=step, t0=step * 4e-9, clock=r["clock"])
    rel = np.zeros(out.n)
    for g in (("x", "y", "z"), ("vx", "vy", "vz")):
        d = np.sqrt(sum((getattr(out, k) - ost[k]) ** 2 for k in g))
        rel = np.maximum(rel, d / np.sqrt(sum(ost[k] ** 2 for k in g)))
    assert float(np.mean(rel < 1e-9)) >= 0.99, np.sort(rel)[-5:]
    assert abs(rs["collisions"] - r["collisions"]) <= 0.01 * r["collisions"]
