"""The per-step table of constant-voltage RF and AC drives and the parallel
clock sum, where their rules change: a launch of 16 steps or more reads the
table, a shorter one evaluates the cosines per lane (the same FP64 bits, so
the two splits of a run are equal exactly); the clock is proposed 32 or 256
steps at a time and checked step by step, and must equal the serial sum."""
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


def _ensembles(kind):
    geom = {"origin_m": [0.0, 0.0, -0.025], "length_m": 0.05, "radius_m": 0.004}
    env = {"temperature_K": 300.0, "pressure_Pa": 50.0, "gas_species": "He"}
    rf = {"RF": {"voltage_V": 200.0, "frequency_Hz": 1.0e6}, "DC": {"quad_V": 1.0, "axial_V": 2.0}}
    quad = cfg.ensemble_params({"instrument": "QuadrupoleRF", "geometry": geom, "env": env, "fields": rf}, 1e-18, 1e-9)
    trap = cfg.ensemble_params({"instrument": "LQIT", "geometry": geom, "env": env, "fields": rf}, 1e-18, 1.7e-9)
    trap.update(ac_dipolar=1, ac_amplitude_V=(0.5, 0.25), ac_frequency_Hz=(1.1e5, 1.3e5), ac_phase_rad=(0.0, 0.5),
                ac_ramp=(1.0, 1.0))
    ac = dict(trap, rf_voltage_V=0.0, dc_quad_V=0.0)
    ims = cfg.ensemble_params({"instrument": "IMS", "geometry": geom, "env": env, "fields": {"DC": {"EN_Td": 5.0}}},
                              1e-18, 1e-9)
    return {"quad": [quad], "trap": [trap], "ac": [ac], "mixed": [ims, trap, quad]}[kind]


@pytest.mark.parametrize("integrator", [capi.INTEGRATOR_BORIS, capi.INTEGRATOR_RK4])
@pytest.mark.parametrize("kind", ["quad", "trap", "ac", "mixed"])
@pytest.mark.parametrize("steps", [16, 17, 130])
def test_table_and_lane_cosines_give_the_same_fp64_run(kind, steps, integrator):
    ens = _ensembles(kind)
    n = 70
    spec = cfg.species_spec(n * len(ens), 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                            {"type": "thermal", "temperature_K": 300.0})
    st = generate_ions(3, [spec])
    off = np.arange(len(ens) + 1, dtype=np.uint64) * n
    out = []
    for per_launch in (0, 15):             # one launch with the table; launches of 15 without
        with Simulation(ens, precision=capi.PREC_FP64, integrator=integrator, collision=capi.COLLISION_HSS,
                        rng_seed=9, steps_per_launch=per_launch) as sim:
            sim.upload(st, ens_offsets=off)
            sim.set_clock(0, np.full(len(ens), 3.1e-7))
            rs = sim.advance(steps)
            out.append((sim.download(), rs, sim.clock()[1]))
    (a, ra, ta), (b, rb, tb) = out
    for k in ("x", "y", "z", "vx", "vy", "vz", "active", "t_death"):
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k))
    assert ra["collisions"] == rb["collisions"]
    np.testing.assert_array_equal(ta, tb)


@pytest.mark.parametrize("steps", [1, 2, 31, 33, 63, 64, 65, 255, 256, 257, 1000, 5000])
@pytest.mark.parametrize("t0,dt", [(0.0, 5e-10), (0.0, 2.0 ** -30), (1.0, 1e-9), (3e-7, 1.7e-9), (1e-3, 3.0 * 2.0 ** -60),
                                   (0.7, 1e-30)])
def test_clock_is_the_serial_sum(t0, dt, steps):
    e = _ensembles("mixed")[0]
    e = dict(e, dt_s=dt)
    st = generate_ions(3, [cfg.species_spec(3, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                            {"type": "thermal", "temperature_K": 300.0})])
    with Simulation([e, dict(e, dt_s=3 * dt)], precision=capi.PREC_MIXED, collision=capi.COLLISION_NONE) as sim:
        sim.upload(st, ens_offsets=np.array([0, 1, 3], dtype=np.uint64))
        sim.set_clock(7, np.array([t0, t0 + dt]))
        sim.advance(steps)
        step, t = sim.clock()
    want = []
    for a, d in ((t0, dt), (t0 + dt, 3 * dt)):
        for _ in range(steps):
            a = a + d
        want.append(a)
    assert step == 7 + steps
    np.testing.assert_array_equal(t, want)


def test_caller_capture_of_an_rf_run_replays():
    """icb_advance captured into the caller's graph (no table: a longer later
    launch may replace it) and replayed, with such a launch in between, equals
    the same steps advanced directly."""
    import torch
    ens = _ensembles("trap")
    st = generate_ions(3, [cfg.species_spec(200, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                            {"type": "thermal", "temperature_K": 300.0})])
    out = []
    for captured in (False, True):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream), \
                Simulation(ens, precision=capi.PREC_FP64, collision=capi.COLLISION_HSS, rng_seed=9) as sim:
            sim.set_stream(stream.cuda_stream)
            sim.upload(st)
            sim.advance(20)
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    sim.advance_async(40)
                g.replay()
                sim.advance(600)
                g.replay()
            else:
                sim.advance(40)
                sim.advance(600)
                sim.advance(40)
            sim.synchronize()
            out.append(sim.download())
            torch.cuda.synchronize()
    for k in ("x", "y", "z", "vx", "vy", "vz", "active"):
        np.testing.assert_array_equal(getattr(out[0], k), getattr(out[1], k))
