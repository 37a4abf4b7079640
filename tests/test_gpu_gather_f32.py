"""The single-precision gather (two lanes per ion, sixteen ions per warp) at
the sizes where its grouping can go wrong: fewer ions than a warp holds, one
more and one less than a warp's and a block's ions, ions in the mesh's
corners (neighbour columns cut by the mesh), excluded ions between others,
and cutoffs from under one cell to several (the table form of the long-range
term as well as the polynomial).

Tolerance: positions enter as floats relative to the mesh origin (error
2^-24 of the 12 mm box, 7e-10 m) and the ions sit on a lattice jittered to
keep at least 0.1 mm between neighbours, so a pair's 1/r^2 field is off by at
most 2 * 2 * 7e-10 / 1e-4 = 3e-5 of itself; the mesh and the sums add float
rounding below that.  1e-4 of the RMS field bounds it, as in the solver's
other single-precision tests."""
from __future__ import annotations

import numpy as np
import pytest

import p3m
from icarion_b200 import _capi as capi
from icarion_b200.sim import Simulation, device_count
from test_gpu_spacecharge import _field_free, _state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _lattice(n, lo, hi, seed):
    """n ions on a 0.3 mm lattice jittered by +-0.1 mm, half of them in a
    dense lump and the rest spread over the whole box."""
    rng = np.random.default_rng(seed)
    g = [np.arange(l + 2e-4, u - 6e-4, 3e-4) for l, u in zip(lo, hi)]
    pts = np.stack(np.meshgrid(*g, indexing="ij"), axis=-1).reshape(-1, 3)
    near = np.argsort(((pts - (lo + 0.3 * (hi - lo))) ** 2).sum(1), kind="stable")
    take = np.concatenate([near[:(n + 1) // 2], rng.choice(near[(n + 1) // 2:], n // 2, replace=False)])
    p = pts[rng.permutation(take)] + rng.uniform(-1e-4, 1e-4, (n, 3))
    q = np.where(rng.random(n) < 0.2, -1.0, 1.0) * 1.602176634e-19
    return p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), q


@pytest.mark.parametrize("cutoff,alpha", [(2.0, 1.0), (0.7, 2.5), (3.4, 1.0)])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 257])
def test_gather_matches_oracle_at_group_edges(n, cutoff, alpha):
    mesh = (20, 16, 12)
    lo, hi = np.array([-6e-3, -4.8e-3, -3.6e-3]), np.array([6e-3, 4.8e-3, 3.6e-3])
    h = (hi - lo) / np.array(mesh)
    x, y, z, q = _lattice(n, lo, hi, seed=n)
    act = np.ones(n, dtype=np.uint8)
    act[3::11] = 0
    want = p3m.p3m_field(x, y, z, q, act, lo, h, mesh, alpha / h.max(), cutoff * h.max())
    with Simulation([_field_free()], precision=capi.PREC_MIXED, collision=capi.COLLISION_NONE, rng_seed=1) as sim:
        sim.upload(_state(x, y, z, q, act))
        sim.configure_space_charge(capi.SC_P3M_ISOLATED, mesh, lo, hi, alpha_h=alpha, pp_cutoff_cells=cutoff)
        got = sim.space_charge_field()
    rms = np.sqrt(np.mean(np.sum(want ** 2, axis=0)))
    assert np.max(np.abs(got - want)) <= 1e-4 * rms
    assert np.all(got[:, act == 0] == 0.0)


def test_an_excluded_ion_without_a_position_changes_nothing():
    """Four ions share a group of slots: an excluded one that holds no number
    must add exactly nothing to the others in its group."""
    mesh = (20, 16, 12)
    lo, hi = np.array([-6e-3, -4.8e-3, -3.6e-3]), np.array([6e-3, 4.8e-3, 3.6e-3])
    x, y, z, q = _lattice(30, lo, hi, seed=3)
    act = np.ones(30, dtype=np.uint8)
    act[[4, 11, 20]] = 0
    fields = []
    for bad in (False, True):
        if bad:
            x[4], y[11], z[20] = np.nan, np.inf, -np.inf
        with Simulation([_field_free()], precision=capi.PREC_MIXED, collision=capi.COLLISION_NONE, rng_seed=1) as sim:
            sim.upload(_state(x, y, z, q, act))
            sim.configure_space_charge(capi.SC_P3M_ISOLATED, mesh, lo, hi, alpha_h=1.0, pp_cutoff_cells=2.0)
            fields.append(sim.space_charge_field())
    assert np.all(np.isfinite(fields[1]))
    assert np.array_equal(fields[0], fields[1])
