"""icb_advance without statistics on handles whose fields depend on time through
constant-voltage RF or AC drives only: it enqueues, whatever the launch length
and however little device memory is left (their drive table is sized at the
upload; without the memory for it the lanes evaluate the cosines, with the
same FP64 bits)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200.sim import Simulation, device_count, generate_ions
from test_gpu_rf_table import _ensembles

pytestmark = pytest.mark.gpu

SLEEP = 200_000_000          # clock cycles: at least 0.1 s
STATE = ("x", "y", "z", "vx", "vy", "vz", "active", "t_death")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _ions(n):
    return generate_ions(3, [cfg.species_spec(n, 200.0 * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
                                              {"type": "gaussian", "center": [0, 0, 0], "std": [2e-4] * 3},
                                              {"type": "thermal", "temperature_K": 300.0})])


def _advance_while_busy(sim, stream, steps):
    """Whether each advance returned with the work ahead of it still running."""
    ahead = []
    for k in steps:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(SLEEP)
            slept = stream.record_event()
        sim.advance_async(k)
        ahead.append(not slept.query())
        sim.synchronize()
    return ahead


def _run(ens, steps, per_ens=40, per_launch=0, clear_wave=False):
    st = _ions(per_ens * len(ens))
    off = np.arange(len(ens) + 1, dtype=np.uint64) * per_ens
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1000)
    with Simulation(ens, precision=capi.PREC_FP64, collision=capi.COLLISION_HSS, rng_seed=9,
                    steps_per_launch=per_launch) as sim:
        sim.set_stream(stream.cuda_stream)
        if clear_wave:
            sim.set_waveform(0, 0, _constant(2.0))
        sim.upload(st, ens_offsets=off)
        if clear_wave:
            sim.set_waveform(0, 0, None)
        ahead = _advance_while_busy(sim, stream, steps)
        return ahead, sim.download()


def _constant(v):
    w = capi.Waveform()
    w.type = 0
    w.p[0] = v
    return w


@pytest.mark.parametrize("clear_wave", [False, True])
@pytest.mark.parametrize("kind", ["quad", "trap", "ac", "mixed"])
def test_growing_launches_only_enqueue(kind, clear_wave):
    steps = [15, 16, 40, 600, 1700]
    ens = _ensembles(kind)
    _run(ens, steps)                      # kernels loaded
    ahead, out = _run(ens, steps, clear_wave=clear_wave and kind == "quad")
    assert all(ahead), ahead
    _, want = _run(ens, steps, per_launch=15)
    for k in STATE:
        np.testing.assert_array_equal(getattr(out, k), getattr(want, k))


def test_run_without_memory_for_the_table():
    """256 quadrupoles of 16,384 steps a launch: a 436 MB table, 256 MB left."""
    ens = _ensembles("quad") * 256
    steps = [40, 20, 600]
    _, want = _run(ens, steps, per_ens=2, per_launch=16384)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    fill = torch.empty(free - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        ahead, out = _run(ens, steps, per_ens=2, per_launch=16384)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert all(ahead), ahead
    for k in STATE:
        np.testing.assert_array_equal(getattr(out, k), getattr(want, k))
