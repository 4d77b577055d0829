"""The work a model has this framework do, as timed cases.

Every case is a dict of plain values with a ``kind``:

* ``step``      one ``Microphysics.__call__`` (plain FP64 or mixed form);
* ``ensemble``  one batched ``MicrophysicsEnsemble.step`` of four domains;
* ``physics``   ``DycoreToPhysics`` then ``Physics.__call__``: the physics of
                one model step, from the dycore's fields to the updated ones;
* ``update``    ``UpdateAtmosphereState.__call__``: the way back to the dycore;
* ``winds``     ``agrid_to_dgrid_tiles``: the wind tendencies of 1 to 6 tiles
                onto the D grid;
* ``vjp``       ``step_vjp``: the adjoint of one microphysics step;
* ``window``    ``rollout`` through ``torch.autograd``: a short window of
                steps forward and backward, as a 4-D assimilation runs it.

``nx`` x ``ny`` columns of ``nz`` levels; a "cN" case is the six N x N tiles
of a cubed sphere side by side (N x 6N), the layout bench.py uses. Inputs are
drawn on the GPU with the distributions of ``pyshield_b200.inputs``. Fields
are NDSL storages: three halo points, one extra point a dimension, i fastest.
"""

import math
import types

import torch

H = 3  # halo points
PTOP = 100.0  # model top [Pa]
TENDENCIES = ("pt_dt", "qv_dt", "ql_dt", "qr_dt", "qi_dt", "qs_dt", "qg_dt", "qa_dt", "udt", "vdt")
STATE = ("pt", "qvapor", "qliquid", "qrain", "qice", "qsnow", "qgraupel", "qcld", "ua", "va", "delprsi", "delz", "wmp")
# physical constants of the model (SI units)
GRAV, RDGAS, RVGAS, CP_AIR = 9.80665, 287.05, 461.50, 1004.6
ZVIR, KAPPA = RVGAS / RDGAS - 1.0, RDGAS / CP_AIR
C_ICE, C_LIQ, CV_AIR, CV_VAP = 1972.0, 4.1855e3, CP_AIR - RDGAS, 3.0 * RVGAS


def listed():
    return [
        # the smallest call: one C12 tile, where launch and host latency count
        {"name": "step_tile12_l79", "kind": "step", "precision": "plain", "nx": 12, "ny": 12, "nz": 79, "dt": 150.0, "sedi_heat": False},
        # the headline benchmark: the whole C96 sphere
        {"name": "step_c96_l79", "kind": "step", "precision": "plain", "nx": 96, "ny": 576, "nz": 79, "dt": 180.0, "sedi_heat": False},
        # a rank's ragged subdomain at the deep vertical grid, with sedimentation heating, two sub-steps
        {"name": "step_ragged_l127_heat", "kind": "step", "precision": "plain", "nx": 53, "ny": 61, "nz": 127, "dt": 225.0, "sedi_heat": True},
        # the mixed form on the headline domain, and at the deep vertical grid
        {"name": "step_c96_l79_mixed", "kind": "step", "precision": "mixed", "nx": 96, "ny": 576, "nz": 79, "dt": 180.0, "sedi_heat": False},
        {"name": "step_c48_l127_mixed", "kind": "step", "precision": "mixed", "nx": 48, "ny": 288, "nz": 127, "dt": 180.0, "sedi_heat": False},
        # an ensemble of domains of different sizes and steps in one launch
        {"name": "ensemble_mixed_l79", "kind": "ensemble", "precision": "mixed", "n1": 24, "n2": 48, "n3": 31, "n4": 17, "nz": 79, "dt": 150.0},
        # a model's physics step: the whole C96 sphere, and a small ragged rank
        {"name": "physics_c96_l79", "kind": "physics", "precision": "plain", "nx": 96, "ny": 576, "nz": 79, "dt": 150.0},
        {"name": "physics_ragged_l63", "kind": "physics", "precision": "plain", "nx": 37, "ny": 29, "nz": 63, "dt": 150.0},
        # the tendencies and tracers back into the dycore's columns, then its D-grid winds
        {"name": "update_c96_l79", "kind": "update", "nx": 96, "ny": 576, "nz": 79, "dt": 150.0},
        {"name": "winds_c96_six_tiles", "kind": "winds", "n": 96, "tiles": 6, "nz": 79, "dt": 150.0},
        # the adjoint: one step's VJP, and a window through torch.autograd
        {"name": "vjp_c48_l79", "kind": "vjp", "nx": 48, "ny": 288, "nz": 79, "dt": 150.0},
        {"name": "window_c24_l79", "kind": "window", "nx": 24, "ny": 144, "nz": 79, "dt": 150.0, "steps": 4},
    ]


def draw(rng):
    """One more case of the same ranges: 144 to 55,296 columns (fewer where
    a column costs more), 31 to 127 levels, steps of 90 to 300 s."""
    kind = rng.choice(("step", "step", "step", "physics", "update", "winds", "vjp", "window", "ensemble"))
    nz = rng.choice((79, rng.randint(31, 64), rng.randint(65, 96), rng.randint(97, 127)))
    dt = float(rng.randint(90, 300))
    if kind == "winds":
        return {"kind": kind, "n": rng.randint(12, 96), "tiles": rng.randint(1, 6), "nz": min(nz, 79), "dt": dt}
    if kind == "ensemble":
        sizes = {f"n{m}": rng.randint(8, 48) for m in (1, 2, 3, 4)}
        return {"kind": kind, "precision": rng.choice(("plain", "mixed")), **sizes, "nz": max(65, nz), "dt": dt}
    most = {"step": 55296, "physics": 55296, "update": 55296, "vjp": 13824, "window": 3456}[kind] * 79 // nz
    if kind in ("vjp", "window"):
        dt = float(rng.randint(90, 150))  # one sub-step, as the listed ones
    elif dt >= 225.0:
        most //= 2  # two sub-steps
    ncol = int(math.exp(rng.uniform(math.log(144), math.log(most))))
    nx = rng.randint(8, max(9, min(128, int(math.sqrt(ncol)))))
    case = {"kind": kind, "nx": nx, "ny": max(1, ncol // nx), "nz": nz, "dt": dt}
    if kind == "window":
        case["steps"] = rng.randint(1, 4)
    if kind in ("step", "physics"):
        case["precision"] = rng.choice(("plain", "mixed"))
    if kind == "step":
        case["sedi_heat"] = rng.random() < 0.25
    return case


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _normal(g, sigma, shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64) * sigma


def _columns(nx, ny, nz, seed):
    """Seeded columns as (nx, ny, nz) fields in i-fastest memory, (nx, ny)
    land: hybrid levels under a random surface pressure, a lapse-rate
    profile with noise, RH U(0.3, 1.05), condensate where it can exist."""
    g = _gen(seed)
    s2, s3 = (ny, nx), (nz, ny, nx)
    ps = _uniform(g, 980.0e2, 1030.0e2, s2)
    s = (torch.arange(nz + 1, device="cuda", dtype=torch.float64) / nz) ** 1.7
    pe = PTOP + (ps - PTOP) * s[:, None, None]
    delp, lnr, p_mid = pe[1:] - pe[:-1], torch.log(pe[1:] / pe[:-1]), 0.5 * (pe[1:] + pe[:-1])
    ts = _uniform(g, 280.0, 302.0, s2)
    noise = _normal(g, 1.5, s3)
    t = torch.empty(s3, device="cuda", dtype=torch.float64)
    z = torch.zeros(s2, device="cuda", dtype=torch.float64)
    for k in range(nz - 1, -1, -1):
        h = RDGAS * torch.clamp(ts - 6.5e-3 * z, min=215.0) / GRAV * lnr[k]
        t[k] = torch.clamp(ts - 6.5e-3 * (z + 0.5 * h), min=215.0) + noise[k]
        z = z + RDGAS * t[k] / GRAV * lnr[k]
    es = 611.21 * torch.exp((-2339.5 * torch.log(t / 273.16) + 3.139057e6 * (t - 273.16) / (t * 273.16)) / RVGAS)
    qsat = RDGAS / RVGAS * es / torch.clamp(p_mid - (1.0 - RDGAS / RVGAS) * es, min=1.0)
    rh = _uniform(g, 0.3, 1.05, s3)
    qv = torch.clamp(rh * qsat, max=0.05)
    warm = t > 273.16

    def condensate(lo, hi, where):
        return torch.where(where, torch.exp(_uniform(g, math.log(lo), math.log(hi), s3)), 0.0)

    f = {"pt": t, "qvapor": qv, "qliquid": condensate(1e-7, 2e-3, (rh > 0.9) & (t > 253.0)),
         "qrain": condensate(1e-7, 1e-3, warm)}
    for name in ("qice", "qsnow", "qgraupel"):
        f[name] = condensate(1e-8, 5e-4, ~warm)
    cond = sum(f[q] for q in ("qliquid", "qrain", "qice", "qsnow", "qgraupel"))
    f["qcld"] = (cond > 1e-6).double()
    f["ua"], f["va"] = _normal(g, 10.0, s3), _normal(g, 10.0, s3)
    f["delprsi"] = delp.contiguous()
    f["delz"] = -RDGAS * t * (1.0 + ZVIR * qv) / GRAV * lnr
    f["wmp"] = _normal(g, 1.0, s3)
    fields = {k: v.permute(2, 1, 0) for k, v in f.items()}
    return fields, (_uniform(g, 0.0, 1.0, s2) < 0.3).double().t()


def _storage(nx, ny, nz, inner=None, fill=0.0):
    """An NDSL storage (nx + 2H + 1, ny + 2H + 1, nz + 1), i fastest, holding ``inner`` in the compute domain."""
    shape = (nx + 2 * H + 1, ny + 2 * H + 1) + ((nz + 1,) if nz else ())
    a = torch.full(shape[::-1], fill, device="cuda", dtype=torch.float64).permute(*reversed(range(len(shape))))
    if inner is not None:
        box = (slice(H, H + nx), slice(H, H + ny)) + ((slice(0, nz),) if nz else ())
        a[box] = inner
    return a


def _q(a, nx, ny, nz, interface=False):
    from pyshield_b200.quantity import Quantity

    if a.dim() == 2:
        return Quantity(a, ("x", "y"), "", (H, H), (nx, ny))
    return Quantity(a, ("x", "y", "z"), "", (H, H, 0), (nx, ny, nz + interface))


def _area(nx, ny):
    n = max(1, int(round(math.sqrt(nx * ny / 6.0))))  # the cell of a cubed sphere with as many columns
    return _storage(nx, ny, 0, fill=4.0 * math.pi * 6.3712e6 ** 2 / (6.0 * n * n))


def _grid(nx, ny, nz):
    from pyshield_b200.grid import GridData, GridIndexing, QuantityFactory, StencilFactory

    gi = GridIndexing(nx, ny, nz, H)
    return StencilFactory(gi), QuantityFactory(gi), GridData(_q(_area(nx, ny), nx, ny, 0), PTOP)


def _config(case):
    from pyshield_b200._config import PhysicsConfig

    return PhysicsConfig(dt_atmos=case["dt"], do_sedi_heat=bool(case.get("sedi_heat", False)))


def _mp_state(nx, ny, nz, seed):
    """A MicrophysicsState of seeded columns with zero tendencies."""
    from pyshield_b200.microphysics import MicrophysicsState

    f, land = _columns(nx, ny, nz, seed)
    q = {k: _q(_storage(nx, ny, nz, v), nx, ny, nz) for k, v in f.items()}
    zero = _q(_storage(nx, ny, nz), nx, ny, nz)
    return MicrophysicsState(
        **{k: q[k] for k in STATE}, delp=q["delprsi"], omga=zero, dz=zero, tendency=zero,
        land=_q(_storage(nx, ny, 0, land), nx, ny, 0))


def _columns_of(case):
    """The columns of a differentiated step: plain (nx, ny, nz) tensors."""
    f, land = _columns(case["nx"], case["ny"], case["nz"], case["seed"])
    x = [f[k] for k in STATE]
    x.append(_storage(case["nx"], case["ny"], case["nz"])[:case["nx"], :case["ny"], :case["nz"]].clone())  # qaz
    return x, land.t().contiguous().t()


def _physics_inputs(nx, ny, nz, seed):
    """The dycore's 16 fields and the physics state's own storages."""
    g = _gen(seed + 1)
    f, land = _columns(nx, ny, nz, seed)
    s3 = (nx, ny, nz)
    f["delp"] = f.pop("delprsi")
    f.pop("wmp")
    f["qo3mr"], f["qsgs_tke"] = _uniform(g, 1e-8, 1e-5, s3), _uniform(g, 0.0, 2.0, s3)
    f["w"], f["omga"] = _uniform(g, -1.0, 1.0, s3), _uniform(g, -2.0, 2.0, s3)
    # the halo holds a neighbour's plausible temperature, thickness and height
    fill = {"pt": 260.0, "delp": 1000.0, "delz": -300.0}
    dycore = {k: _storage(nx, ny, nz, v, fill.get(k, 0.0)) for k, v in f.items()}
    for k in ("delp", "delz"):
        dycore[k][..., nz] = 0.0
    prsi = PTOP + 1000.0 * torch.arange(nz + 1, device="cuda", dtype=torch.float64)
    phii = GRAV * 300.0 * torch.arange(nz, -1, -1, device="cuda", dtype=torch.float64)
    physics = {k: v.clone() for k, v in dycore.items()}
    for k in ("specific_humidity", "qliquid", "qice", "qrain", "qsnow", "qgraupel", "cloud_fraction", "pt", "ua", "va"):
        physics["physics_updated_" + k] = _storage(nx, ny, nz)
    for k in ("delprsi", "phil", "dz", "wmp", "prsik"):
        physics[k] = _storage(nx, ny, nz)
    physics["prsi"] = _storage(nx, ny, nz) + prsi
    physics["phii"] = _storage(nx, ny, nz) + phii
    physics["land"] = _storage(nx, ny, 0, land)
    return dycore, physics


UPDATE_DYCORE = ("qvapor", "qliquid", "qrain", "qsnow", "qice", "qgraupel")
UPDATE_PHYSICS = ("specific_humidity", "qliquid", "qrain", "qsnow", "qice", "qgraupel")


def _update_inputs(nx, ny, nz, seed):
    """The storages of the way back: the dycore's fields, the physics state
    a step later, and the tendencies the dycore accumulates."""
    g = _gen(seed + 1)
    f, _ = _columns(nx, ny, nz, seed)
    s3 = (nx, ny, nz)
    d = {k: _storage(nx, ny, nz, f[k]) for k in UPDATE_DYCORE + ("pt", "ua", "va")}
    d["delp"] = _storage(nx, ny, nz, f["delprsi"], 1000.0)
    for k in ("pe", "peln", "pk"):
        d[k] = _storage(nx, ny, nz)
    d["pe"][..., 0] = PTOP
    d["ps"] = _storage(nx, ny, 0)
    p = {"ua": d["ua"].clone(), "va": d["va"].clone(), "pt": d["pt"].clone()}
    for k, n in zip(UPDATE_DYCORE, UPDATE_PHYSICS):
        # a step's change of a few per cent; a few points below zero, which the fill mends
        change = 1.0 + _normal(g, 0.02, s3)
        p["physics_updated_" + n] = _storage(nx, ny, nz, f[k] * change - 1e-9 * (_uniform(g, 0.0, 1.0, s3) < 0.01))
    for k, sigma in (("ua", 0.1), ("va", 0.1), ("pt", 0.05)):
        p["physics_updated_" + k] = _storage(nx, ny, nz, f[k] + _normal(g, sigma, s3))
    prsi = _storage(nx, ny, nz)
    prsi[H:H + nx, H:H + ny, 0] = PTOP
    prsi[H:H + nx, H:H + ny, 1:] = PTOP + torch.cumsum(f["delprsi"], 2)
    p["prsi"] = prsi
    t = {k: _storage(nx, ny, nz, _normal(g, 1e-4, s3)) for k in ("u_dt", "v_dt")}
    t["pt_dt"] = _storage(nx, ny, nz)
    return d, p, t


def _wind_inputs(case, seed):
    """Per tile: the winds, the tendencies with a filled halo, the geometry."""
    n, nz, g = case["n"], case["nz"], _gen(seed)
    s2, s3 = (n + 2 * H + 1, n + 2 * H + 1), (nz + 1, n + 2 * H + 1, n + 2 * H + 1)
    tiles = []
    for _ in range(case["tiles"]):
        a = {k: _normal(g, 10.0, s3).permute(2, 1, 0) for k in ("u", "v")}
        a.update({k: _normal(g, 1e-3, s3).permute(2, 1, 0) for k in ("u_dt", "v_dt")})
        for name in ("vlon", "vlat", "es1_", "ew2_"):
            v = _normal(g, 1.0, (3,) + s2)
            v = v / v.norm(dim=0)  # unit vectors
            a.update({f"{name}{m + 1}": v[m].t() for m in range(3)})
        for e in "we":
            a["edge_vect_" + e] = _uniform(g, 0.0, 1.0, s2).t()
        for e in "sn":
            a["edge_vect_" + e] = _uniform(g, 0.0, 1.0, s2[:1])
        tiles.append(a)
    return tiles


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    case = dict(case, seed=seed)
    return {"step": _prepare_step, "ensemble": _prepare_ensemble, "physics": _prepare_physics,
            "update": _prepare_update, "winds": _prepare_winds, "vjp": _prepare_vjp, "window": _prepare_window}[kind](case)


def _prepare_step(case):
    from pyshield_b200.microphysics import Microphysics

    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mp = Microphysics(*_grid(nx, ny, nz), _config(case), precision=case["precision"])
    return {"case": case, "mp": mp, "state": _mp_state(nx, ny, nz, case["seed"])}


def _prepare_ensemble(case):
    from pyshield_b200.ensemble import MicrophysicsEnsemble

    sizes = [case[f"n{m}"] for m in (1, 2, 3, 4)]
    states = [_mp_state(n, 6 * n, case["nz"], case["seed"] + 100 * m) for m, n in enumerate(sizes)]
    areas = [_q(_area(n, 6 * n), n, 6 * n, 0) for n in sizes]
    steps = [case["dt"] * f for f in (1.0, 0.8, 0.9, 1.0)]
    ens = MicrophysicsEnsemble(_config(case), states, areas, steps, precision=case["precision"])
    ens.autotune()
    return {"case": case, "ens": ens, "states": states}


def _prepare_physics(case):
    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.coupling import DycoreToPhysics
    from pyshield_b200.physics import Physics, PhysicsState

    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    sf, qf, gd = _grid(nx, ny, nz)
    cfg = PhysicsConfig(dt_atmos=case["dt"], npz=nz)
    dycore, physics = _physics_inputs(nx, ny, nz, case["seed"])
    q = {k: _q(v, nx, ny, nz, k in ("phii", "prsi", "prsik")) for k, v in physics.items()}
    ps = PhysicsState(**q, quantity_factory=qf, schemes=cfg.schemes)
    return {"case": case, "ps": ps, "physics": Physics(sf, qf, gd, cfg, precision=case["precision"]),
            "d2p": DycoreToPhysics(sf, qf, cfg, False, False),
            "dycore": types.SimpleNamespace(**{k: _q(v, nx, ny, nz) for k, v in dycore.items()})}


def _prepare_update(case):
    from pyshield_b200._config import PhysicsConfig
    from pyshield_b200.coupling import UpdateAtmosphereState

    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    d, p, t = ({k: _q(v, nx, ny, nz) for k, v in part.items()} for part in _update_inputs(nx, ny, nz, case["seed"]))
    sf, _, gd = _grid(nx, ny, nz)
    return {"case": case, "dycore": types.SimpleNamespace(**d), "physics": types.SimpleNamespace(**p), "tend": t,
            "update": UpdateAtmosphereState(sf, gd, PhysicsConfig(dt_atmos=case["dt"]))}


def _prepare_winds(case):
    from pyshield_b200.dwind import AGrid2DGridPhysics

    n, nz = case["n"], case["nz"]
    calls = []
    for a in _wind_inputs(case, case["seed"]):
        sf, qf, _ = _grid(n, n, nz)
        gi = sf.grid_indexing
        gi.south_edge = gi.north_edge = gi.west_edge = gi.east_edge = True
        w = {k: _q(a.pop(k), n, n, nz) for k in ("u", "v", "u_dt", "v_dt")}
        namelist = types.SimpleNamespace(dt_atmos=case["dt"], npx=n + 1, npy=n + 1, layout=(1, 1))
        whole = types.SimpleNamespace(subtile_index=lambda rank: (0, 0))
        a2d = AGrid2DGridPhysics(sf, qf, whole, 0, namelist, types.SimpleNamespace(grid_type=0, **a))
        calls.append((a2d, w["u"], w["v"], w["u_dt"], w["v_dt"]))
    return {"case": case, "calls": calls}


def _cotangents(case, seed):
    """A cotangent for each output of a step, in the output's own memory order."""
    g = _gen(seed + 2)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    c3 = [_normal(g, 1.0, (nz, ny, nx)).permute(2, 1, 0) for _ in range(12)]
    return c3 + [_normal(g, 1.0, (ny, nx)).t() for _ in range(4)]


def _prepare_vjp(case):
    from pyshield_b200.microphysics import Microphysics

    mp = Microphysics(*_grid(case["nx"], case["ny"], case["nz"]), _config(case))
    x, land = _columns_of(case)
    return {"case": case, "mp": mp, "x": x, "land": land, "cot": _cotangents(case, case["seed"])}


def _prepare_window(case):
    s = _prepare_vjp(case)
    g = _gen(case["seed"] + 2)
    # the cotangent of the final state: the misfit to an analysis
    s["cot"] = [_normal(g, 1.0, t.permute(2, 1, 0).shape).permute(2, 1, 0) for t in s["x"]]
    return s


# --------------------------------------------------------------------- run
def run(s):
    return {"step": _run_step, "ensemble": _run_ensemble, "physics": _run_physics, "update": _run_update,
            "winds": _run_winds, "vjp": _run_vjp, "window": _run_window}[s["case"]["kind"]](s)


def _step_outputs(state):
    return {k: getattr(state, k).view for k in TENDENCIES + ("wmp",)}


def _run_step(s):
    mp = s["mp"]
    mp(s["state"], s["case"]["dt"])
    return {**_step_outputs(s["state"]), "rain": mp.rain, "snow": mp.snow, "ice": mp.ice, "graupel": mp.graupel}


def _run_ensemble(s):
    s["ens"].step()
    return [{**_step_outputs(st), "precip": list(s["ens"].precip(m))} for m, st in enumerate(s["states"])]


PRESTEP_OUT = ("qvapor", "qliquid", "qice", "qrain", "qsnow", "qgraupel", "qo3mr", "qsgs_tke", "delp", "pt", "delprsi",
               "phii", "phil", "prsi", "dz")
PHYSICS_OUT = PRESTEP_OUT + ("wmp",) + tuple(
    "physics_updated_" + k for k in ("specific_humidity", "qliquid", "qice", "qrain", "qsnow", "qgraupel",
                                     "cloud_fraction", "pt", "ua", "va"))


def _run_physics(s):
    s["d2p"](s["dycore"], s["ps"])
    s["physics"](s["ps"], s["case"]["dt"])
    mp = s["ps"].microphysics
    return {**{k: getattr(s["ps"], k).view for k in PHYSICS_OUT}, **{k: getattr(mp, k).view for k in TENDENCIES}}


UPDATE_OUT = UPDATE_DYCORE + ("delp", "pt", "pe", "peln", "pk")


def _run_update(s):
    u, d, p, t = s["update"], s["dycore"], s["physics"], s["tend"]
    u(d, p, t["u_dt"], t["v_dt"], t["pt_dt"], s["case"]["dt"])
    return {**{k: getattr(d, k).data for k in UPDATE_OUT}, **{k: v.data for k, v in t.items()}, "ps": d.ps.data,
            "filled": p.physics_updated_specific_humidity.data, "u_srf": u.u_srf, "v_srf": u.v_srf}


def _run_winds(s):
    from pyshield_b200.dwind import agrid_to_dgrid_tiles

    agrid_to_dgrid_tiles(s["calls"])
    return [{"u": u.data, "v": v.data, "u_dt": u_dt.data, "v_dt": v_dt.data} for _, u, v, u_dt, v_dt in s["calls"]]


def _run_vjp(s):
    from pyshield_b200.adjoint import step_vjp

    return step_vjp(s["mp"], s["x"], s["land"], s["cot"], s["case"]["dt"])


def _run_window(s):
    from pyshield_b200.adjoint import STATE as NAMES
    from pyshield_b200.adjoint import rollout

    x = [t.detach().requires_grad_(True) for t in s["x"]]
    final, _ = rollout(s["mp"], dict(zip(NAMES, x)), s["land"], s["case"]["dt"], s["case"]["steps"])
    # delprsi and delz pass through a step unchanged
    grads = torch.autograd.grad([final[k] for k in NAMES], x, s["cot"])
    return {"final": [final[k].detach() for k in NAMES], "grads": list(grads)}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: each input field read once, each output written once. The
    operations of the microphysics depend on which processes each point
    meets, so none are counted."""
    nz, kind = case["nz"], case["kind"]

    def step_bytes(ncol):
        # 24 fields in (13 state, 10 tendencies, the cloud-fraction accumulator), 12 out; land, area, 4 totals
        return ncol * (36 * nz + 6) * 8

    if kind == "ensemble":
        return {"bytes": sum(step_bytes(6 * case[f"n{m}"] ** 2) for m in (1, 2, 3, 4)), "flops": 0}
    if kind == "winds":
        n = case["n"]
        points = 2 * (n * n + 4 * n) + 4 * n * (n + 1) + 2 * (n + 2) ** 2  # tendencies, u and v twice, zeroed points
        return {"bytes": case["tiles"] * 8 * (nz * points + 6 * (n * n + 4 * n) + 6 * n * (n + 1)), "flops": 0}
    nx, ny = case["nx"], case["ny"]
    ncol, full = nx * ny, (nx + 2 * H) * (ny + 2 * H)
    if kind == "step":
        return {"bytes": step_bytes(ncol), "flops": 0}
    if kind == "physics":
        # the dycore's 16 fields in; out: those 16, eight new physics fields, the tendencies and the updated state
        return {"bytes": 8 * (nz * (16 * ncol + 34 * ncol + 28 * ncol) + 5 * nz * (full - ncol)), "flops": 0}
    if kind == "update":
        return {"bytes": 8 * (full * 3 * nz + ncol * 36 * (nz + 1)), "flops": 0}
    # the adjoint: 14 inputs and 12 cotangents in, 14 gradients out
    one = ncol * (40 * nz + 6) * 8
    if kind == "vjp":
        return {"bytes": one, "flops": 0}
    # a step forward: 14 fields in, 12 out, and the advanced state (10 fields read, written)
    return {"bytes": case["steps"] * (one + ncol * 46 * nz * 8), "flops": 0}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The coupling stencils in plain torch FP64. The microphysics and its
    adjoint have no value besides their own FP64 results."""
    kind = case["kind"]
    if kind == "physics":
        return _exact_physics(case, seed)
    if kind == "update":
        return _exact_update(case, seed)
    if kind == "winds":
        return [_exact_wind_tile(a, case) for a in _wind_inputs(case, seed)]
    return None


def _exact_physics(case, seed):
    """What the pre-steps leave (DycoreToPhysics' copy, statein, get_prs_fv3,
    get_phi_fv3, prepare_microphysics); None for what the microphysics writes."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    d, _ = _physics_inputs(nx, ny, nz, seed)
    box = (slice(H, H + nx), slice(H, H + ny), slice(0, nz))
    f = {k: v[box].contiguous() for k, v in d.items()}
    zero = torch.zeros((nx, ny, 1), device="cuda", dtype=torch.float64)
    phii = torch.cat([torch.flip(torch.cumsum(torch.flip(-f["delz"] * GRAV, (2,)), 2), (2,)), zero], 2)
    tracers = ("qvapor", "qliquid", "qrain", "qice", "qsnow", "qgraupel", "qo3mr")
    q = {k: f[k] * f["delp"] for k in tracers}
    dm = f["delp"] - q["qliquid"] - q["qrain"] - q["qice"] - q["qsnow"] - q["qgraupel"]
    prsi = torch.cat([zero + PTOP, PTOP + torch.cumsum(dm, 2)], 2)
    q = {k: v / dm for k, v in q.items()}
    tv = f["pt"] * (1.0 + ZVIR * torch.clamp(q["qvapor"], min=1e-10))
    layer = phii[..., :-1] - phii[..., 1:]
    delp = torch.maximum(torch.minimum(dm * RDGAS * tv / layer, prsi[..., 1:] - 0.01 * dm), prsi[..., :-1] + 0.01 * dm)
    phi = torch.cat([torch.flip(torch.cumsum(torch.flip(layer, (2,)), 2), (2,)), zero], 2)
    out = dict.fromkeys(PHYSICS_OUT + TENDENCIES)
    out.update(q, qsgs_tke=f["qsgs_tke"] / dm, delp=delp, pt=f["pt"], delprsi=prsi[..., 1:] - prsi[..., :-1],
               phii=phi, phil=0.5 * (2.0 * phi[..., 1:] + layer), prsi=prsi, dz=(phi[..., 1:] - phi[..., :-1]) / GRAV)
    return out


def _fill(delp, q):
    """fill_gfs_delp: vapour borrowed upwards, floored, borrowed downwards."""
    q, nk, low = q.clone(), q.shape[2], 1e-9
    for k in range(nk - 2, -1, -1):
        q[..., k] += torch.where(q[..., k + 1] < low, (q[..., k + 1] - low) * delp[..., k + 1] / delp[..., k], 0.0)
    q[..., 1:] = torch.clamp(q[..., 1:], min=low)
    for k in range(1, nk):
        q[..., k] += torch.where(q[..., k - 1] < 0.0, q[..., k - 1] * delp[..., k - 1] / delp[..., k], 0.0)
    return torch.clamp(q, min=0.0)


def _exact_update(case, seed):
    nx, ny, nz, dt = case["nx"], case["ny"], case["nz"], case["dt"]
    d, p, t = _update_inputs(nx, ny, nz, seed)
    full = (slice(0, nx + 2 * H), slice(0, ny + 2 * H), slice(0, nz))
    filled = p["physics_updated_specific_humidity"]
    filled[full] = _fill(d["delp"][full], filled[full])
    ij = (slice(H, H + nx), slice(H, H + ny))
    c = ij + (slice(0, nz),)
    prsi = p["prsi"][ij]
    dp = prsi[..., 1:] - prsi[..., :-1]
    mass = {k: dp * p["physics_updated_" + n][c] for k, n in zip(UPDATE_DYCORE, UPDATE_PHYSICS)}
    delp = d["delp"][c] * (1.0 - sum(d[k][c] for k in UPDATE_DYCORE)) + sum(mass.values())
    for a, b in (("u_dt", "ua"), ("v_dt", "va"), ("pt_dt", "pt")):
        t[a][c] += (p["physics_updated_" + b][c] - p[b][c]) / dt
    d["delp"][c] = delp
    for k, v in mass.items():
        d[k][c] = v / delp
    # moist_cv on all nz + 1 levels
    q = {k: d[k][ij] for k in UPDATE_DYCORE}
    liquid, solid = q["qliquid"] + q["qrain"], q["qice"] + q["qsnow"] + q["qgraupel"]
    cvm = (1.0 - (q["qvapor"] + liquid + solid)) * CV_AIR + q["qvapor"] * CV_VAP + liquid * C_LIQ + solid * C_ICE
    d["pt"][ij] += t["pt_dt"][ij] * dt * CP_AIR / cvm
    t["pt_dt"][ij] = 0.0
    pe = d["pe"][ij]
    pe[..., 1:] = pe[..., :1] + torch.cumsum(delp, 2)
    d["peln"][ij][..., 1:] = torch.log(pe[..., 1:])
    d["pk"][ij][..., 1:] = pe[..., 1:] ** KAPPA
    d["ps"][ij] = pe[..., nz]
    return {**{k: d[k] for k in UPDATE_OUT}, **t, "ps": d["ps"], "filled": filled,
            "u_srf": d["ua"][ij][..., nz - 1], "v_srf": d["va"][ij][..., nz - 1]}


def _exact_wind_tile(a, case):
    n, nz, dt5 = case["n"], case["nz"], 0.5 * case["dt"]
    mid = n // 2 + 2
    ks, lo, hi = slice(0, nz), H - 1, H + n + 1
    v3 = [a["u_dt"][..., ks] * a[f"vlon{m}"][..., None] + a["v_dt"][..., ks] * a[f"vlat{m}"][..., None] for m in (1, 2, 3)]
    p = slice(lo, hi)
    ue, ve = [torch.zeros_like(v) for v in v3], [torch.zeros_like(v) for v in v3]
    for x, y, v in zip(ue, ve, v3):
        x[p, p] = v[p, lo - 1:hi - 1] + v[p, p]
        y[p, p] = v[lo - 1:hi - 1, p] + v[p, p]
    # the corrections on the tile's edges read the neighbour towards the middle
    along = torch.arange(H, H + n, device="cuda")
    nbr = torch.where(along <= mid, along + 1, along - 1)
    for y in ve:
        for line, e in ((H, a["edge_vect_w"]), (H + n, a["edge_vect_e"])):
            w, old = e[line, along][:, None], y[line].clone()
            y[line, along] = w * old[nbr] + (1.0 - w) * old[along]
    for x in ue:
        for line, e in ((H, a["edge_vect_s"]), (H + n, a["edge_vect_n"])):
            w, old = e[along][:, None], x[:, line].clone()
            x[along, line] = w * old[nbr] + (1.0 - w) * old[along]
    c, c1 = slice(H, H + n), slice(H, H + n + 1)
    a["u"][c, c1, ks] += dt5 * sum(ue[m][c, c1] * a[f"es1_{m + 1}"][c, c1, None] for m in range(3))
    a["v"][c1, c, ks] += dt5 * sum(ve[m][c1, c] * a[f"ew2_{m + 1}"][c1, c, None] for m in range(3))
    for k in ("u_dt", "v_dt"):
        a[k][p, p, ks] = 0.0
    return {k: a[k] for k in ("u", "v", "u_dt", "v_dt")}
