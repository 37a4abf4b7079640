"""The buffers that icb_spacecharge_set_peers grows: they are ready when the
call returns, for a next solve on another stream (icb_set_stream does not
wait)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from icarion_b200 import _capi as capi
from icarion_b200 import fticr
from icarion_b200.sim import Simulation, device_count

pytestmark = pytest.mark.gpu

N = 2000


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _sim(precision, stream):
    """A cloud whose field bound is given, so that setting peers solves nothing."""
    cell = fticr.fticr_cell(n_ions=N, mesh=32)
    sim = Simulation([cell.ensemble], precision=precision, collision=capi.COLLISION_NONE, rng_seed=1)
    sim.set_stream(stream.cuda_stream)
    sim.upload(cell.ions)
    sim.configure_space_charge(capi.SC_P3M_ISOLATED, [32] * 3, cell.sc_box_min, cell.sc_box_max, field_bound=1e4)
    return sim


def _peers(sim, n):
    """This handle's own ions once more, then n - N rows without charge."""
    buf = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    sim.spacecharge_export(buf.data_ptr())
    sim.synchronize()
    torch.cuda.synchronize()
    return buf


@pytest.mark.parametrize("precision", [capi.PREC_MIXED, capi.PREC_FP64])
def test_solve_on_another_stream_after_growth(precision):
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    fields = []
    for streams in ((a, a, a), (a, b, a)):
        with _sim(precision, streams[0]) as sim:
            got = []
            for n, s in zip((N + 1, 8_000_001), streams[1:]):
                buf = _peers(sim, n)
                sim.set_spacecharge_peers(buf.data_ptr(), n)
                assert a.query() and b.query()
                sim.set_stream(s.cuda_stream)
                got.append(sim.space_charge_field())
            fields.append(got)
    for whole, switched in zip(*fields):
        np.testing.assert_array_equal(whole, switched)
    assert np.max(np.abs(fields[0][0])) > 0


def _fill(leave):
    """All but `leave` bytes of the device's free memory."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info(0)[0] - leave, dtype=torch.uint8, device="cuda")


def test_peers_that_do_not_fit_are_refused_and_the_handle_goes_on():
    """20 M peers need 1.7 GB of buffers, 512 MB are left."""
    s = torch.cuda.Stream()
    with _sim(capi.PREC_MIXED, s) as sim:
        want = sim.space_charge_field()
        buf = _peers(sim, N + 1)
        fill = _fill(512 << 20)
        try:
            with pytest.raises(RuntimeError):
                sim.set_spacecharge_peers(buf.data_ptr(), 20_000_000)
            with pytest.raises(RuntimeError, match="could not be had"):
                sim.space_charge_field()
            with pytest.raises(RuntimeError):
                sim.advance(1)
            sim.set_spacecharge_peers(0, 0)
            np.testing.assert_array_equal(sim.space_charge_field(), want)
        finally:
            del fill
            torch.cuda.empty_cache()
        sim.set_spacecharge_peers(buf.data_ptr(), N + 1, 0, N + 1)
        np.testing.assert_array_equal(sim.space_charge_field(), want)
        assert sim.advance(2)["steps"] == 2


@pytest.mark.parametrize("precision", [capi.PREC_MIXED, capi.PREC_FP64, capi.PREC_MIXED_HILO])
def test_ions_that_do_not_fit_are_refused_and_the_handle_goes_on(precision):
    """4 M ions need over 400 MB, 256 MB are left; the ions uploaded before
    are gone with their arrays, and a smaller upload works."""
    cell = fticr.fticr_cell(n_ions=4_000_000, mesh=32)
    small = fticr.fticr_cell(n_ions=N, mesh=32).ions
    with Simulation([cell.ensemble], precision=precision, collision=capi.COLLISION_NONE, rng_seed=1) as sim:
        sim.upload(small)
        sim.advance(10)
        want = sim.download()
        fill = _fill(256 << 20)
        try:
            with pytest.raises(RuntimeError):
                sim.upload(cell.ions)
            for call in (lambda: sim.advance(10), lambda: sim.update_state(cell.ions), sim.moments):
                with pytest.raises(RuntimeError, match="no ions"):
                    call()
            sim.set_clock(0, np.zeros(1))
            sim.upload(small)
            sim.advance(10)
            out = sim.download()
        finally:
            del fill
            torch.cuda.empty_cache()
    for k in ("x", "y", "z", "vx", "vy", "vz", "active"):
        np.testing.assert_array_equal(getattr(out, k), getattr(want, k))
