"""Timed workloads of the batch step, through the public Python mirror of the
C ABI (icarion_b200.sim, .ipm, .fticr, .sweep).

Every case is one thing a program that uses this library does over and over:

    engine    the reference engine's own step order through the plug points
              (host state in, push, collide, finalize, host state out)
    drift     drift-tube ions between two snapshots: advance, download
    host      the engine fast path: host state in, many steps, host state out
    steploop  the per-step kernel, one launch per engine step
    sweep     an E/N sweep of many ensembles in one launch sequence (CUDA graph)
    tims      trapped IMS with a ramped axial profile and RF confinement
    quad      RF quadrupole transmission, no gas, RK4
    trap      linear ion trap with RF, AC drive and buffer gas
    ipm       drift-tube ions with the learned interaction-potential deflection
    fticr     FT-ICR cell with space charge solved every step
    train     training the deflection network

The largest cases return their state through page-locked host memory, as
the benchmark does.  Handles keep their ions between passes: a pass carries
on from where the one before left the cloud.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from icarion_b200 import _capi as capi
from icarion_b200 import config as cfg
from icarion_b200 import fticr, ipm, sweep
from icarion_b200.sim import IonState, Simulation, generate_ions

STATE = ("x", "y", "z", "vx", "vy", "vz")
COUNTS = ("steps", "candidates", "collisions", "rate_overflows", "deaths", "arrivals")
PRECISION = {"fp64": capi.PREC_FP64, "mixed": capi.PREC_MIXED, "hilo": capi.PREC_MIXED_HILO}


def listed() -> list:
    return [
        # the smallest call: a reference engine that keeps its own loop and
        # calls the plug points every step, host state in and out
        {"name": "engine_step_1k", "kind": "engine", "ions": 1024, "steps": 1, "precision": "fp64"},
        # the plain IMS run (4,096 ions, FP64, HSS in N2 at 20 Td), one
        # snapshot interval of 1,000 steps
        {"name": "ims_fp64_4k", "kind": "drift", "ions": 4096, "steps": 1000, "precision": "fp64", "td": 20.0},
        # the mixed-precision IMS run at full size, end to end from host state
        {"name": "ims_mixed_1m", "kind": "host", "ions": 1048576, "steps": 1000, "precision": "mixed", "td": 20.0},
        # an engine with work of its own between steps: every step is one
        # launch that streams the whole state through HBM
        {"name": "step_loop_4m", "kind": "steploop", "ions": 4194304, "steps": 60, "precision": "mixed", "td": 20.0},
        # 64 uneven ensembles, 2-100 Td, three species, one graph launch
        {"name": "en_sweep_64", "kind": "sweep", "ensembles": 64, "count_max": 65536, "steps": 1000},
        # trapped IMS during the elution ramp: a field that changes every step
        {"name": "tims_mixed_256k", "kind": "tims", "ions": 262144, "steps": 500, "precision": "mixed"},
        # quadrupole mass filter, collision free, FP64 RK4 (the reference's
        # accuracy setting for RF fields)
        {"name": "quad_rk4_fp64_20k", "kind": "quad", "ions": 20000, "steps": 500, "precision": "fp64"},
        # ion trap with RF, dipolar AC excitation and helium
        {"name": "trap_mixed_100k", "kind": "trap", "ions": 100001, "steps": 500, "precision": "mixed"},
        # learned interaction-potential collisions at 40 Td
        {"name": "ipm_learned_200k", "kind": "ipm", "ions": 200000, "steps": 500, "td": 40.0},
        # the FT-ICR cell at full size: a P3M solve (128^3 mesh) every step
        {"name": "fticr_262k", "kind": "fticr", "ions": 262144, "steps": 8, "mesh": 128},
        # a small FT-ICR cloud (tuning and validation runs)
        {"name": "fticr_10k", "kind": "fticr", "ions": 10007, "steps": 8, "mesh": 64},
        # training the deflection network on 2^16 samples, one epoch
        {"name": "ipm_train_64k", "kind": "train", "samples": 65536, "batch": 1024, "epochs": 1},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["engine", "drift", "drift", "host", "steploop", "sweep", "tims", "quad", "trap", "ipm",
                       "fticr", "fticr", "train"])
    if kind == "engine":
        return {"kind": kind, "ions": _log_int(rng, 64, 16384), "steps": 1, "precision": rng.choice(["fp64", "mixed"])}
    if kind == "drift":
        return {"kind": kind, "ions": _log_int(rng, 500, 60000), "steps": rng.choice([250, 500, 1000]),
                "precision": rng.choice(["fp64", "mixed"]), "td": round(rng.uniform(5.0, 60.0), 2)}
    if kind == "host":
        return {"kind": kind, "ions": _log_int(rng, 200000, 1048576), "steps": rng.choice([500, 1000]),
                "precision": rng.choice(["mixed", "mixed", "fp64"]), "td": round(rng.uniform(5.0, 40.0), 2)}
    if kind == "steploop":
        return {"kind": kind, "ions": _log_int(rng, 100000, 4194304), "steps": rng.randint(20, 60),
                "precision": rng.choice(["mixed", "mixed", "fp64"]), "td": round(rng.uniform(5.0, 40.0), 2)}
    if kind == "sweep":
        return {"kind": kind, "ensembles": rng.randint(8, 64), "count_max": _log_int(rng, 8000, 65536),
                "steps": rng.choice([500, 1000])}
    if kind == "tims":
        return {"kind": kind, "ions": _log_int(rng, 4000, 262144), "steps": rng.choice([250, 500]),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "quad":
        return {"kind": kind, "ions": _log_int(rng, 1000, 40000), "steps": rng.choice([250, 500]),
                "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "trap":
        return {"kind": kind, "ions": _log_int(rng, 4000, 200000), "steps": rng.choice([250, 500]),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "ipm":
        return {"kind": kind, "ions": _log_int(rng, 20000, 200000), "steps": rng.choice([250, 500]),
                "td": round(rng.uniform(10.0, 80.0), 2)}
    if kind == "fticr":
        return {"kind": kind, "ions": _log_int(rng, 2000, 262144), "steps": rng.randint(2, 8),
                "mesh": rng.choice([64, 96, 128, 128])}
    return {"kind": kind, "samples": _log_int(rng, 8192, 65536), "batch": rng.choice([512, 1000, 1024, 2048]),
            "epochs": 1}


# -- set-ups -------------------------------------------------------------------
def _pinned(n: int, dtype=torch.float64) -> np.ndarray:
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _host_state(st: IonState, times: bool) -> IonState:
    """The ions' host arrays in page-locked memory."""
    out = {}
    for k in STATE:
        out[k] = _pinned(st.n)
        out[k][:] = getattr(st, k)
    act = _pinned(st.n, torch.uint8)
    act[:] = st.active
    death, arrival = (_pinned(st.n), _pinned(st.n)) if times else (None, None)
    return IonState(mass=st.mass, charge=st.charge, active=act, t_death=death, t_arrival=arrival, **out)


def _cloud(seed: int, n: int, mass_da: float, sigma_m: float, center=(0.0, 0.0, 0.0), temperature=300.0) -> IonState:
    return generate_ions(seed, [cfg.species_spec(
        n, mass_da * cfg.AMU_TO_KG, cfg.ELEM_CHARGE_C,
        {"type": "gaussian", "center": list(center), "std": [sigma_m] * 3},
        {"type": "thermal", "temperature_K": temperature})])


def _ims(td: float, pressure: float = 1000.0) -> dict:
    return {"instrument": "IMS", "geometry": {"origin_m": [0.0, 0.0, -0.01], "length_m": 0.1, "radius_m": 0.05},
            "env": {"temperature_K": 300.0, "pressure_Pa": pressure, "gas_species": "N2"},
            "fields": {"DC": {"EN_Td": td}}}


TIMS = {"instrument": "TIMS", "geometry": {"origin_m": [0.0, 0.0, -0.01], "length_m": 0.02, "radius_m": 0.005},
        "env": {"temperature_K": 300.0, "pressure_Pa": 310.0, "gas_species": "N2",
                "flow_model": "axial_uniform", "axial_flow_velocity_m_s": 134.0},
        "fields": {"RF": {"voltage_V": 180.0, "frequency_Hz": 2.0e6}, "DC": {"quad_V": 0.0},
                   "TIMS": {"z_positions_m": [0.0, 0.02], "axial_field_initial_profile_V_m": [0.0, -4495.0],
                            "axial_field_final_profile_V_m": [0.0, 0.0], "ramp_start_s": 1.0e-5,
                            "ramp_end_s": 4.0e-2, "ramp_mode": "linear"}}}
QUAD = {"instrument": "QuadrupoleRF", "geometry": {"origin_m": [0.0, 0.0, -0.05], "length_m": 0.1, "radius_m": 0.005},
        "env": {"temperature_K": 300.0, "pressure_Pa": 1.0, "gas_species": "He"},
        "fields": {"RF": {"voltage_V": 200.0, "frequency_Hz": 1.0e6}, "DC": {"quad_V": 5.0, "axial_V": 1.0}}}
TRAP = {"instrument": "LQIT", "geometry": {"origin_m": [0.0, 0.0, -0.025], "length_m": 0.05, "radius_m": 0.004},
        "env": {"temperature_K": 300.0, "pressure_Pa": 10.0, "gas_species": "He"},
        "fields": {"RF": {"voltage_V": 200.0, "frequency_Hz": 1.0e6}, "DC": {"quad_V": 1.0, "axial_V": 2.0}}}
DT_RF = 1e-9


def _trap_ensemble() -> dict:
    e = cfg.ensemble_params(TRAP, 100e-20, DT_RF)
    e.update(ac_dipolar=1, ac_amplitude_V=(0.5, 0.25), ac_frequency_Hz=(1.1e5, 1.3e5), ac_phase_rad=(0.0, 0.5),
             ac_ramp=(1.0, 1.0))
    return e


def prepare(case: dict, seed: int) -> dict:
    kind, s = case["kind"], {"case": case}
    cloud_seed = 1 + seed % 2000000011
    if kind == "train":
        setup = ipm.IpmSetup()
        s["x"], s["y"], _, _ = ipm.training_set(setup, n=case["samples"], seed=seed)
        s["seed"] = seed
        return s
    if kind in ("engine", "drift", "host", "steploop"):
        td = case.get("td", 20.0)
        st = _cloud(cloud_seed, case["ions"], 200.0, 5e-4)
        ens = [cfg.ensemble_params(_ims(td), 150e-20, 5e-10, detector_z_m=2.0e-3)]
        sim = Simulation(ens, precision=PRECISION[case["precision"]], collision=capi.COLLISION_HSS, rng_seed=seed,
                         collision_test=capi.TEST_PER_STEP if kind == "steploop" else capi.TEST_CLOCK)
        sim.upload(st)
    elif kind == "sweep":
        sw = sweep.en_sweep(n_ensembles=case["ensembles"], count_max=case["count_max"], count_seed=123,
                            ion_seed=cloud_seed)
        st = sw.ions
        sim = Simulation(sw.ensembles, precision=capi.PREC_MIXED, collision=capi.COLLISION_HSS, rng_seed=seed,
                         use_graphs=1)
        sim.upload(st, ens_offsets=sw.offsets)
    elif kind == "tims":
        st = _cloud(cloud_seed, case["ions"], 200.0, 5e-4)
        sim = Simulation([cfg.ensemble_params(TIMS, 150e-20, 5e-10)], precision=PRECISION[case["precision"]],
                         collision=capi.COLLISION_HSS, rng_seed=seed)
        sim.apply_time_fields(0, TIMS)
        sim.upload(st)
    elif kind == "quad":
        st = _cloud(cloud_seed, case["ions"], 100.0, 2e-4)
        sim = Simulation([cfg.ensemble_params(QUAD, 100e-20, DT_RF)], precision=PRECISION[case["precision"]],
                         integrator=capi.INTEGRATOR_RK4, collision=capi.COLLISION_NONE, rng_seed=seed)
        sim.upload(st)
    elif kind == "trap":
        st = _cloud(cloud_seed, case["ions"], 200.0, 2e-4)
        sim = Simulation([_trap_ensemble()], precision=PRECISION[case["precision"]], collision=capi.COLLISION_HSS,
                         rng_seed=seed)
        sim.upload(st)
    elif kind == "ipm":
        setup = ipm.IpmSetup()
        x, y, _, _ = ipm.training_set(setup, n=1 << 14, seed=2024)
        params, _ = ipm.train(x, y, epochs=8, batch=256, lr=3e-3)
        ens, st, off = ipm.drift_ensembles(setup, (case["td"],), case["ions"], seed=cloud_seed)
        sim = Simulation(ens, precision=capi.PREC_MIXED, collision=capi.COLLISION_IPM_MLP, rng_seed=seed)
        sim.upload(st, ens_offsets=off)
        sim.configure_ipm(setup)
        sim.set_mlp(params)
    elif kind == "fticr":
        cell = fticr.fticr_cell(n_ions=case["ions"], seed=cloud_seed, mesh=case["mesh"])
        st = cell.ions
        sim = Simulation([cell.ensemble], precision=capi.PREC_FP64, collision=capi.COLLISION_LANGEVIN, rng_seed=seed)
        sim.upload(st)
        fticr.configure(sim, cell, solver_fp32=True)
    else:
        raise ValueError(kind)
    s["sim"] = sim
    s["host"] = _host_state(st, times=kind != "host")
    return s


# -- one pass ------------------------------------------------------------------
def _out(host: IonState, stats: dict) -> dict:
    out = {k: getattr(host, k) for k in STATE}
    out["active"] = host.active
    if host.t_death is not None:
        out["t_death"], out["t_arrival"] = host.t_death, host.t_arrival
    out["counts"] = np.array([stats[k] for k in COUNTS], dtype=np.int64)
    return out


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        params, losses = ipm.train(s["x"], s["y"], epochs=case["epochs"], batch=case["batch"], seed=s["seed"])
        return {"params": params, "losses": losses}
    sim, host = s["sim"], s["host"]
    if kind == "engine":
        for _ in range(case["steps"]):
            sim.update_state(host)
            sim.step_batch()
            coll = sim.handle_batch()
            fin = sim.finalize()
            sim.download(into=host)
        return _out(host, {**fin, "candidates": coll["candidates"], "collisions": coll["collisions"]})
    if kind == "host":
        return _out(host, sim.advance_host(host, case["steps"]))
    stats = sim.advance(case["steps"])
    sim.download(into=host)
    return _out(host, stats)


# -- what a pass cannot do without ----------------------------------------------
# Flops of one engine step of one ion: the push (Boris in a uniform field
# 15; with a magnetic field or an RF / trap field about 45; RK4 in an RF
# field about 150), and per accepted collision about 150 for the neutral,
# the acceptance and the scatter.  About 9 % of ion-steps collide at
# dt = 0.1 / nu.  The state crosses HBM once per launch.
PUSH_FLOPS = {"engine": 15, "drift": 15, "host": 15, "steploop": 15, "sweep": 15, "tims": 45, "quad": 150, "trap": 45,
              "ipm": 15, "fticr": 45}
COLL_FLOPS = {"quad": 0.0, "fticr": 0.0, "trap": 2.0, "tims": 4.0, "ipm": 0.09 * (150 + 2 * 4417)}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        n = case["samples"] - case["samples"] % case["batch"]
        # forward 2 x 4417, backward about twice that, per sample
        return {"bytes": 12 * n * case["epochs"] + 2 * 4 * capi.MLP_N_PARAMS, "flops": 6.0 * 4417 * n * case["epochs"]}
    if kind == "sweep":
        lo, hi = 1000.0, float(case["count_max"])
        n = case["ensembles"] * (hi - lo) / math.log(hi / lo)     # mean of a log-uniform count
    else:
        n = case["ions"]
    steps = case["steps"]
    v = 8 if case.get("precision", "mixed") == "fp64" or kind == "fticr" else 4
    state = 2 * (24 + 3 * v) + 1                                  # positions, velocities in and out, flag
    flops = n * steps * (PUSH_FLOPS[kind] + COLL_FLOPS.get(kind, 0.09 * 150))
    launches = steps if kind in ("steploop", "fticr") else 1
    nbytes = n * (state * launches + 48 + 1)                      # and the doubles that come back to the host
    if kind == "fticr":
        # pairs inside the cutoff (2 cells) of a Gaussian cloud of 1 mm, 25
        # flops each; forward and three inverse transforms of the padded mesh
        m = case["mesh"]
        pairs = n * n / (8.0 * math.pi ** 1.5 * 1e-9) * (4.0 / 3.0) * math.pi * (2 * 14e-3 / m) ** 3
        fft = 4 * 2.5 * (2 * m) ** 3 * math.log2((2 * m) ** 3)
        flops += steps * (25.0 * pairs + fft)
        nbytes += steps * 4 * 4 * m ** 3                          # charge and three field components on the mesh
    return {"bytes": float(nbytes), "flops": float(flops)}


# -- 64-bit values ---------------------------------------------------------------
def _field_sum(p: torch.Tensor, q: torch.Tensor, soft: float = 1e-10) -> torch.Tensor:
    """Softened direct Coulomb sum at every ion (the field P3M approximates)."""
    n = p.shape[1]
    e = torch.empty_like(p)
    rows = max(1, min(n, (1 << 28) // n))
    for a in range(0, n, rows):
        d = p[:, a:a + rows, None] - p[:, None, :]
        r2 = (d * d).sum(0)
        w = torch.where(r2 > 0, q / ((r2 + soft * soft) * r2.clamp_min(1e-300).sqrt()), 0.0)
        e[:, a:a + rows] = 8.987551787e9 * (d * w).sum(2)
    return e


def _exact_fticr(case: dict, seed: int):
    cell = fticr.fticr_cell(n_ions=case["ions"], seed=1 + seed % 2000000011, mesh=case["mesh"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    st, ens = cell.ions, cell.ensemble
    p, v = t([st.x, st.y, st.z]), t([st.vx, st.vy, st.vz])
    m, q = t(st.mass), t(st.charge)
    length, radius, dt = ens["length_m"], ens["radius_m"], ens["dt_s"]
    k = ens["radial_V"] / (length ** 2 / 8 + radius ** 2 / 4)
    tz = ens["B_T"][2] * q / m * dt * 0.5
    sz = 2 * tz / (1 + tz * tz)
    for _ in range(case["steps"]):
        e = _field_sum(p, q) + k * torch.stack([p[0], p[1], -2 * (p[2] - length / 2)])
        a = e * q / m
        v = v + a * (dt / 2)
        x1, y1 = v[0] + v[1] * tz, v[1] - v[0] * tz
        v = torch.stack([v[0] + y1 * sz, v[1] - x1 * sz, v[2]])
        p = p + v * dt
        v = v + a * (dt / 2)
    return dict(zip(STATE, [a.cpu().numpy() for a in (*p, *v)]))


def _exact_quad(case: dict, seed: int):
    st = _cloud(1 + seed % 2000000011, case["ions"], 100.0, 2e-4)
    f = QUAD["fields"]
    r0, length = QUAD["geometry"]["radius_m"], QUAD["geometry"]["length_m"]
    w = 2 * math.pi * f["RF"]["frequency_Hz"]
    inv_m = 1.0 / st.mass
    x, v = np.stack([st.x, st.y, st.z]), np.stack([st.vx, st.vy, st.vz])

    def acc(p, t):
        u = f["DC"]["quad_V"] + f["RF"]["voltage_V"] * math.cos(w * t)
        ez = np.full(p.shape[1], f["DC"]["axial_V"] / length)
        return np.stack([-2 * p[0] * u / r0 ** 2, 2 * p[1] * u / r0 ** 2, ez]) * st.charge * inv_m

    t, h = 0.0, DT_RF
    for _ in range(case["steps"]):
        a1 = acc(x, t)
        v2 = v + a1 * (h / 2)
        a2 = acc(x + v * (h / 2), t + h / 2)
        v3 = v + a2 * (h / 2)
        a3 = acc(x + v2 * (h / 2), t + h / 2)
        v4 = v + a3 * h
        a4 = acc(x + v3 * h, t + h)
        x, v = x + (v + 2 * v2 + 2 * v3 + v4) * (h / 6), v + (a1 + 2 * a2 + 2 * a3 + a4) * (h / 6)
        t += h
    return dict(zip(STATE, [*x, *v]))


def exact(case: dict, seed: int):
    """The collision-free cases in plain float64.  The others draw random
    collisions from the library's own counter-based stream, so no value
    exists outside it; training is a chaotic iteration in 32 bits."""
    if case["kind"] == "quad":
        return _exact_quad(case, seed)
    if case["kind"] == "fticr" and case["ions"] * case["ions"] * case["steps"] <= 6e11:
        return _exact_fticr(case, seed)
    return None
