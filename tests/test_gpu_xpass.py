"""The fused x pass of the single-precision mesh at both of its lengths (64-
and 128-node x axes) and at column counts that are no multiple of a block's
(32 or 16), and the neighbouring lengths that keep the separate passes: the
mesh part of the field (cutoff 1/100 cell) within 1e-5 of the oracle's RMS
field, the bound the 128-node case has (float transforms)."""
from __future__ import annotations

import numpy as np
import pytest

import p3m
from icarion_b200 import _capi as capi
from test_gpu_spacecharge import _cloud, _sim, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(64, 25, 20), (64, 16, 8), (64, 9, 33), (128, 9, 12), (63, 16, 8), (65, 8, 16)])
def test_mesh_field_matches_oracle(mesh):
    h = 1e-4
    hi = 0.5 * h * np.array(mesh)
    lo = -hi
    x, y, z, q = _cloud(2000, seed=7, sigma=2e-4)
    act = np.ones(2000, dtype=np.uint8)
    hs = (hi - lo) / np.array(mesh)
    want = p3m.p3m_field(x, y, z, q, act, lo, hs, mesh, 1.0 / hs.max(), 0.01 * hs.max())
    with _sim(_state(x, y, z, q), precision=capi.PREC_MIXED) as sim:
        sim.configure_space_charge(capi.SC_P3M_ISOLATED, mesh, lo, hi, pp_cutoff_cells=0.01)
        got = sim.space_charge_field()
        assert np.array_equal(got, sim.space_charge_field())
    rms = np.sqrt(np.mean(np.sum(want ** 2, axis=0)))
    assert np.max(np.abs(got - want)) <= 1e-5 * rms
