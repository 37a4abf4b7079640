"""The drive table of constant-voltage RF and AC drives in the float forms: the
same launches with the table and with the lanes' own cosines (a run captured
by its caller has no table) give the same bits.  The float lanes evaluate
cos(w t) and a cos(w t + phase) in double, the phase sum contracted, and round
once; the table holds those floats."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200.sim import Simulation, device_count, generate_ions
from test_gpu_rf_table import _ensembles

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


@pytest.mark.parametrize("precision,integrator,collision",
                         [(capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_HSS),
                          (capi.PREC_MIXED, capi.INTEGRATOR_BORIS, capi.COLLISION_NONE),
                          (capi.PREC_MIXED, capi.INTEGRATOR_RK4, capi.COLLISION_HSS),
                          (capi.PREC_MIXED_HILO, capi.INTEGRATOR_BORIS, capi.COLLISION_HSS)])
@pytest.mark.parametrize("kind", ["quad", "trap", "ac", "mixed"])
@pytest.mark.parametrize("steps", [16, 130])
def test_table_and_lane_cosines_give_the_same_float_run(steps, kind, precision, integrator, collision):
    ens = _ensembles(kind)
    n = 300
    st = generate_ions(3, [cfg.species_spec(n * len(ens), 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                            {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                            {"type": "thermal", "temperature_K": 300.0})])
    off = np.arange(len(ens) + 1, dtype=np.uint64) * n
    out = []
    for captured in (False, True):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream), \
                Simulation(ens, precision=precision, integrator=integrator, collision=collision, rng_seed=9) as sim:
            sim.set_stream(stream.cuda_stream)
            sim.upload(st, ens_offsets=off)
            sim.set_clock(0, np.full(len(ens), 3.1e-7))
            sim.advance(3)
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    sim.advance_async(steps)
                for _ in range(3):
                    g.replay()
            else:
                for _ in range(3):
                    sim.advance_async(steps)
            sim.synchronize()
            out.append(sim.download())
            torch.cuda.synchronize()
    for k in ("x", "y", "z", "vx", "vy", "vz", "active", "t_death"):
        np.testing.assert_array_equal(getattr(out[0], k), getattr(out[1], k), err_msg=k)
