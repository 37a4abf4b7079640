"""The staging of the float forms between the caller's doubles and the working
arrays: three arrays where memory allows, one where it does not.  4 M ions of
the mixed forms hold 472 MB with one and 532 MB with three."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import config0_ensemble, config0_ions
from icarion_b200 import _capi as capi
from icarion_b200.sim import Simulation, device_count

pytestmark = pytest.mark.gpu

N = 4_000_000
STATE = ("x", "y", "z", "vx", "vy", "vz", "active")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _sim(precision):
    return Simulation([config0_ensemble()], precision=precision, collision=capi.COLLISION_NONE, rng_seed=1)


def _equal(a, b):
    for k in STATE:
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=k)


@pytest.mark.parametrize("precision", [capi.PREC_MIXED, capi.PREC_MIXED_HILO])
def test_one_staging_array_serves_where_three_do_not_fit(precision):
    st = config0_ions(N)
    with _sim(precision) as sim:
        sim.upload(st)
        sim.advance(5)
        mid = sim.download()
        want = mid.copy()
        sim.advance_host(want, 5, n_chunks=4)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info(0)[0] - (502 << 20), dtype=torch.uint8, device="cuda")
    with _sim(precision) as sim:
        try:
            sim.upload(st)
            sim.advance(5)
            out = sim.download()
            _equal(out, mid)
            if precision == capi.PREC_MIXED:              # the hi/lo form does not overlap its copies
                with pytest.raises(RuntimeError):
                    sim.advance_host(out.copy(), 5, n_chunks=4)
                _equal(sim.download(), mid)
        finally:
            del fill
            torch.cuda.empty_cache()
        sim.advance_host(out, 5, n_chunks=4)
        _equal(out, want)
        _equal(sim.download(), want)
