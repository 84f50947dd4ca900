"""Workloads by which this framework's speed is judged: right-hand sides and time steps of every
equation system, through the public package.

Two calls make up a simulation.  `rhs` evaluates the right-hand side of a state that is resident on
the GPU (what an external time integrator calls every stage); `steps` is a whole run segment: the
state from pinned host memory, Runge-Kutta steps under the CFL condition, the new state back.  A
program builds its handle once and starts many states on it, so handles are kept between states.

`exact` is a plain torch restatement of the discretisation in 64 bits: flux differencing as a full
two-point table per line, logarithmic means by atanh, fluxes of full states.
"""
import importlib.util
import json
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "trixiatmo_gb300"
    if name not in sys.modules:
        folder = os.path.join(_ROOT, "trixiatmo.jl_gb300")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---- the cases ----------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one right-hand side of a test-sized dry mesh (latency and launches)
        dict(name="dry_rhs_tiny", system="dry2d", op="rhs", nx=8, ny=4, polydeg=3),
        # the dry warm bubble of the buoyancy elixirs, one mesh, a run segment
        dict(name="dry_bubble_run", system="dry2d", op="steps", nx=64, ny=32, polydeg=3, steps=20,
             method="CarpenterKennedy2N54"),
        # an ensemble of such bubbles in one handle
        dict(name="dry_ensemble_run", system="dry2d", op="steps", nx=64, ny=32, polydeg=3, steps=2,
             members=64, method="CarpenterKennedy2N54"),
        # the global atmosphere on the cubed-sphere shell, the largest right-hand side
        dict(name="shell_rhs", system="dry3d", op="rhs", trees=16, layers=8, polydeg=5),
        # a run segment on a coarse shell of lower degree
        dict(name="shell_run", system="dry3d", op="steps", trees=8, layers=5, polydeg=3, steps=4,
             method="CarpenterKennedy2N54"),
        # global circulation in potential temperature (flux_tec with the Souza gravity term)
        dict(name="pt_shell_rhs", system="pt3d", op="rhs", trees=8, layers=4, polydeg=4,
             volume="tec", gravity="souza"),
        # inertia-gravity waves in potential temperature, the elixir's 60 x 8 mesh, SSPRK43
        dict(name="pt_waves_run", system="pt2d", op="steps", nx=60, ny=8, polydeg=3, steps=20,
             volume="tec", gravity="waruszewski", method="SSPRK43"),
        # a wide ragged mesh with the entropy- and energy-conserving flux
        dict(name="pt_wide_rhs", system="pt2d", op="rhs", nx=253, ny=67, polydeg=4,
             volume="etec", gravity="artiano"),
        # moist bubble: cloud water, phase change, pressure walls
        dict(name="moist_run", system="moist2d", op="steps", nx=128, ny=64, polydeg=4, steps=2,
             method="CarpenterKennedy2N54"),
        # precipitation bubble with the saturation Newton limiter after every stage
        dict(name="rainy_run", system="rainy2d", op="steps", nx=128, ny=64, polydeg=3, steps=2,
             method="CarpenterKennedy2N54"),
        # shallow water on the cubed sphere, weak form
        dict(name="swe_run", system="swe", op="steps", trees=30, polydeg=3, members=1, steps=10,
             form="weak", method="CarpenterKennedy2N54"),
        # an uneven shallow-water ensemble in the entropy-conserving split form
        dict(name="swe_ensemble_run", system="swe", op="steps", trees=20, polydeg=0, members=12,
             steps=2, form="ec", method="CarpenterKennedy2N54"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    system = rng.choice(["dry2d", "dry2d", "dry3d", "pt2d", "pt3d", "moist2d", "rainy2d", "swe"])
    case = dict(system=system, op=rng.choice(["rhs", "steps"]))
    if system in ("dry3d", "pt3d"):
        case["polydeg"] = rng.choice([2, 3, 4, 5, 7])
        elements = _log_int(rng, 48, 2_000_000 / (case["polydeg"] + 1) ** 3 / (
            1 if case["op"] == "rhs" else 8))
        case["layers"] = rng.randint(2, 8)
        case["trees"] = max(2, int(math.sqrt(elements / 6 / case["layers"])))
    elif system == "swe":
        case["op"] = "steps"
        case["members"] = rng.choice([1, 1, 5, 9])
        case["polydeg"] = rng.choice([2, 3, 5, 7]) if case["members"] == 1 else 0
        case["trees"] = rng.randint(4, 40 if case["members"] == 1 else 20)
        case["form"] = rng.choice(["weak", "ec"])
    else:
        case["polydeg"] = rng.choice([1, 2, 3, 4, 5, 7])
        top = {"dry2d": 2_000_000, "pt2d": 1_000_000, "moist2d": 400_000, "rainy2d": 200_000}
        elements = _log_int(rng, 24, top[system] / (case["polydeg"] + 1) ** 2 / (
            1 if case["op"] == "rhs" else 4))
        case["ny"] = max(2, int(math.sqrt(elements) * rng.uniform(0.3, 0.9)))
        case["nx"] = max(3, elements // case["ny"])
        if system == "dry2d" and case["op"] == "steps" and rng.random() < 0.4:
            case["members"] = rng.choice([3, 7, 16])
            case["nx"] = max(3, case["nx"] // case["members"])
    if system.startswith("pt"):
        case["volume"] = rng.choice(["tec", "ec", "etec"])
        case["gravity"] = rng.choice(["waruszewski", "artiano", "souza"])
    if case["op"] == "steps":
        case["steps"] = rng.randint(1, 3)
        case["method"] = ("CarpenterKennedy2N54" if system == "rainy2d" else
                          rng.choice(["CarpenterKennedy2N54", "SSPRK43", "SSPRK33"]))
    return case


_NV = {"dry2d": 5, "dry3d": 6, "pt2d": 5, "pt3d": 6, "moist2d": 6, "rainy2d": 9, "swe": 3}
_STAGES = {"CarpenterKennedy2N54": 5, "SSPRK43": 4, "SSPRK33": 3}
_CFL = 0.5
_LX, _LZ = 20000.0, 10000.0


def _members(case):
    """(trees, polydeg) of the members of a shallow-water case; polydeg 0: uneven."""
    if case["polydeg"]:
        return [(case["trees"], case["polydeg"])] * case["members"]
    return [(max(3, case["trees"] - 3 * (m % 4)), (3, 5, 7)[m % 3]) for m in range(case["members"])]


def _nodes(case):
    s, n = case["system"], case["polydeg"] + 1
    if s == "swe":
        return sum(6 * k * k * (p + 1) ** 2 for k, p in _members(case))
    if s in ("dry3d", "pt3d"):
        return 6 * case["trees"] ** 2 * case["layers"] * n ** 3
    return case["nx"] * case["ny"] * n * n * case.get("members", 1)


def work(case):
    """Per node and stage: the two-point (or nodal) fluxes of its lines, the stage update and the
    surface terms; state read and written, metric terms read, once."""
    dim = 3 if case["system"] in ("dry3d", "pt3d") else 2
    nv, n = _NV[case["system"]], case["polydeg"] + 1 if case["polydeg"] else 6
    pair = {"dry2d": 55, "dry3d": 75, "pt2d": 55, "pt3d": 70, "moist2d": 85, "rainy2d": 95,
            "swe": 26}[case["system"]]
    evals = 1 if case["op"] == "rhs" else case["steps"] * _STAGES[case["method"]]
    nodes = _nodes(case)
    flops = nodes * evals * (dim * 0.5 * (n - 1) * pair + 12 * nv + 60)
    if case["system"] == "rainy2d" and case["op"] == "steps":
        flops += nodes * evals * 150  # one saturation Newton update
    metric = (16 if case["system"] == "swe" else dim * dim + 1)
    per_eval = 8 * (2 * nv + metric + (0 if case["op"] == "rhs" else 2 * nv))
    return {"bytes": nodes * (evals * per_eval + (0 if case["op"] == "rhs" else 16 * nv)),
            "flops": flops}


# ---- handles ------------------------------------------------------------------------------------
_kept = {}


def _semi(case):
    """The handle a program keeps: one at a time, for any number of states."""
    key = json.dumps({k: v for k, v in case.items() if k not in ("name", "op", "steps", "method")},
                     sort_keys=True)
    if key not in _kept:
        for old in _kept.values():
            old.close()
        _kept.clear()
        _kept[key] = _build(case)
    return _kept[key]


def _build(case):
    tg = _package()
    system, N = case["system"], case["polydeg"]
    if system == "swe":
        return _build_swe(tg, case)
    terms = {"waruszewski": tg.flux_nonconservative_waruszewski_etal,
             "artiano": tg.flux_nonconservative_artiano_etal,
             "souza": tg.flux_nonconservative_souza_etal}
    lmars = (tg.FluxLMARS(340.0), tg.flux_zero)
    wall, source = tg.boundary_condition_slip_wall, None
    if system in ("dry3d", "pt3d"):
        gravity = tg.EARTH_GRAVITATIONAL_ACCELERATION
        mesh = tg.P4estMeshCubedSphereTopography(case["trees"], case["layers"], _RADIUS, _HEIGHT,
                                                 polydeg=N, geometry_on_device=True)
        if system == "dry3d":
            eq = tg.CompressibleEulerEnergyEquationsWithGravity3D(c_p=1004, c_v=717, gravity=gravity)
            vf = (tg.flux_ranocha, terms["waruszewski"])
        else:
            eq = tg.CompressibleEulerPotentialTemperatureEquationsWithGravity3D(
                c_p=1004, c_v=717, gravity=gravity)
            vf = (getattr(tg, "flux_" + case["volume"]), terms[case["gravity"]])
        solver = tg.DGSEM(N, lmars, tg.VolumeIntegralFluxDifferencing(vf))
        return tg.SemidiscretizationHyperbolic(
            mesh, eq, None, solver, source_terms=tg.source_terms_coriolis,
            boundary_conditions={"inside": wall, "outside": wall})
    surface = lmars
    if system == "dry2d":
        eq = tg.CompressibleEulerEnergyEquationsWithGravity2D(c_p=1004, c_v=717, gravity=9.81)
        vf = (tg.flux_ranocha, terms["waruszewski"])
    elif system == "pt2d":
        eq = tg.CompressibleEulerPotentialTemperatureEquationsWithGravity2D(
            c_p=1004, c_v=717, gravity=9.81)
        vf = (getattr(tg, "flux_" + case["volume"]), terms[case["gravity"]])
    elif system == "moist2d":
        eq = tg.CompressibleMoistEulerEquations2D(c_pd=1004, c_vd=717, c_pv=1885, c_vv=1424,
                                                  gravity=9.81)
        vf, surface, source = tg.flux_chandrashekar, tg.FluxLMARS(360.0), tg.source_terms_moist_bubble
    else:
        eq = tg.CompressibleRainyEulerEquations2D()
        vf, surface, source = tg.flux_ec_rain, tg.flux_lax_friedrichs, tg.source_terms_rainy
        wall = tg.boundary_condition_simple_slip_wall
    mesh = tg.StructuredMesh((case["nx"], case["ny"]), (0.0, 0.0), (_LX, _LZ),
                             periodicity=(True, False))
    solver = tg.DGSEM(N, surface, tg.VolumeIntegralFluxDifferencing(vf))
    walls = {"y_neg": wall, "y_pos": wall}
    members = case.get("members", 1)
    if members > 1:
        return tg.SemidiscretizationEnsemble([mesh] * members, eq, [None] * members, solver,
                                             boundary_conditions=walls)
    return tg.SemidiscretizationHyperbolic(mesh, eq, None, solver, source_terms=source,
                                           boundary_conditions=walls)


def _build_swe(tg, case):
    cv = tg.covariant
    if case["form"] == "ec":
        eq = cv.SplitCovariantShallowWaterEquations2D(_GRAVITY, _OMEGA)
        surface = (cv.FluxPlusDissipation(cv.flux_ec, cv.DissipationLocalLaxFriedrichs()),
                   cv.flux_nonconservative_surface_simplified)
        volume = tg.VolumeIntegralFluxDifferencing((cv.flux_ec, cv.flux_nonconservative_ec))
    else:
        eq = cv.CovariantShallowWaterEquations2D(_GRAVITY, _OMEGA)
        surface, volume = tg.flux_lax_friedrichs, tg.VolumeIntegralWeakForm()
    meshes = [cv.P4estMeshCubedSphere2D(k, _RADIUS, polydeg=p) for k, p in _members(case)]
    solvers = [tg.DGSEM(p, surface, volume) for _, p in _members(case)]
    if len(meshes) == 1:
        return tg.SemidiscretizationHyperbolic(
            meshes[0], eq, None, solvers[0], source_terms=cv.source_terms_geometric_coriolis)
    return tg.SemidiscretizationCovariantEnsemble(
        meshes, eq, [None] * len(meshes), solvers, source_terms=cv.source_terms_geometric_coriolis)


# ---- states -------------------------------------------------------------------------------------
_RADIUS, _HEIGHT, _GRAVITY, _OMEGA = 6.37122e6, 30000.0, 9.80616, 7.292e-5
_CP, _CV, _P0 = 1004.0, 717.0, 1.0e5
_R, _GAMMA = _CP - _CV, _CP / _CV
_K = _P0 * (_R / _P0) ** _GAMMA  # p = K rho_theta^gamma


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _initial_state(case, semi, seed):
    """A seeded state on the GPU, [elements, nodes..., variables] (shallow water: flat)."""
    rng = np.random.default_rng(seed)
    system = case["system"]
    if system == "swe":
        return _dev(_swe_state(case, semi, rng))
    x = _dev(semi.node_coordinates)
    if system in ("dry3d", "pt3d"):
        return _shell_state(system, x, rng)
    members = case.get("members", 1)
    per = semi.nelements // members
    return torch.cat([_box_state(system, x[m * per:(m + 1) * per], rng) for m in range(members)])


def _box_state(system, x, rng):
    """A neutral atmosphere (300 K) with a warm bubble of seeded place and strength and a wind."""
    g = 9.81
    xc, zc, amp = rng.uniform(6e3, 14e3), rng.uniform(1.5e3, 4e3), rng.uniform(0.5, 3.0)
    wind = rng.uniform(-15, 15)
    z = x[..., 1]
    r = torch.sqrt((x[..., 0] - xc) ** 2 + (z - zc) ** 2) / 2000.0
    bump = torch.where(r < 1, torch.cos(0.5 * math.pi * r.clamp(max=1.0)) ** 2, 0.0)
    theta = 300.0 + amp * bump
    p = _P0 * (1 - (_R / _CP) * g * z / (_R * 300.0)) ** (_CP / _R)
    T = theta * (p / _P0) ** (_R / _CP)
    rho = p / (_R * T)
    v1 = wind + 3.0 * torch.sin(2 * math.pi * x[..., 0] / _LX + rng.uniform(0, 6))
    v2 = 2.0 * bump * torch.sin(math.pi * z / _LZ)
    kin = 0.5 * (v1 * v1 + v2 * v2)
    if system == "dry2d":
        return torch.stack([rho, rho * v1, rho * v2, rho * (_CV * T + kin), g * z], -1)
    if system == "pt2d":
        return torch.stack([rho, rho * v1, rho * v2, (p / _K) ** (1 / _GAMMA), g * z], -1)
    if system == "moist2d":
        qv = 6e-3 * torch.exp(-z / 3000.0) * (1 + 0.2 * bump)
        ql = 4e-4 * bump + 1e-5
        qd = 1 - qv - ql
        e = (qd * 717.0 + qv * 1424.0 + ql * 4186.0) * T + qv * 3147620.0 + kin
        return torch.stack([rho, rho * v1, rho * v2, rho * e, rho * qv, rho * ql], -1)
    # the rainy state: random humidity, a saturated bubble, some cloud and rain everywhere; slots
    # 7-9 hold the constructed vapour, cloud and temperature (the limiter finds the equilibrium)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 31)))

    def uniform(a, b):
        return a + (b - a) * torch.rand(z.shape, generator=gen, device="cuda", dtype=torch.float64)

    T = 288.0 - 0.0065 * z
    p = _P0 * (T / 288.0) ** (9.80616 / (287.0 * 0.0065))
    rh = torch.where(r <= 1, 1.0, uniform(0.2, 1.0))
    rv = rh * _saturation_pressure(T) / (461.0 * T)
    rd = (p - rv * 461.0 * T) / (287.0 * T)
    rc, rr = uniform(0, 1e-3) * rd, uniform(0, 1e-3) * rd
    e = (717.0 * rd + 1424.0 * rv + 4186.0 * (rc + rr)) * T + rv * 2.5e6
    zero = torch.zeros_like(T)
    return torch.stack([rd, rv + rc, rr, zero, zero, e, rv, rc, T], -1)


def _shell_state(system, x, rng):
    """An isothermal atmosphere in a zonal wind with seeded density bumps."""
    T = rng.uniform(240.0, 260.0)
    r = x.norm(dim=-1)
    rr = r.clamp(min=_RADIUS)
    p = _P0 * torch.exp(_GRAVITY * (_RADIUS ** 2 / rr - _RADIUS) / (_R * T))
    unit = x / r[..., None]
    bump = torch.zeros_like(r)
    for c in rng.normal(size=(4, 3)):
        angle = torch.arccos((unit @ _dev(c / np.linalg.norm(c))).clamp(-1, 1))
        bump += torch.exp(-(angle * 12.0) ** 2)
    rho = p / (_R * T) * (1 + 1e-2 * bump)
    wind = rng.uniform(10, 30)
    v = [-wind * unit[..., 1], wind * unit[..., 0], 5.0 * bump * unit[..., 2]]
    phi = _GRAVITY * (_RADIUS - _RADIUS ** 2 / rr)
    last = (p / (_GAMMA - 1) + 0.5 * rho * sum(w * w for w in v) if system == "dry3d"
            else (p / _K) ** (1 / _GAMMA))
    return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], last, phi], -1)


def _swe_state(case, semi, rng):
    """Geostrophic balance with a seeded Gaussian height bump, in contravariant components."""
    tg = _package()
    cv = tg.covariant

    def start(x, t, eq, amp, c):
        p = cv.initial_condition_geostrophic_balance(x, t, eq)
        d2 = ((x / np.sqrt((x ** 2).sum(-1, keepdims=True)) - c) ** 2).sum(-1)
        p[..., 0] *= 1 + amp * np.exp(-d2 / 0.05)
        return p

    parts = []
    for m in range(case["members"]):
        c = rng.normal(size=3)
        amp, c = rng.uniform(0.01, 0.05), c / np.linalg.norm(c)
        ic = cv.transform_initial_condition(
            lambda x, t, eq, amp=amp, c=c: start(x, t, eq, amp, c), semi.equations)
        parts.append(np.asarray(ic(semi._H.xyz[m], 0.0, semi._H.aux[m])).ravel())
    return np.concatenate(parts)


def prepare(case, seed):
    semi = _semi(case)
    u = _initial_state(case, semi, seed).contiguous()
    state = {"case": case, "semi": semi}
    if case["op"] == "rhs":
        state.update(u=u, du=torch.zeros_like(u))
        torch.cuda.synchronize()
    else:
        state.update(start=u.cpu().pin_memory().numpy().reshape(semi.shape),
                     out=torch.zeros(u.shape, dtype=u.dtype).pin_memory().numpy().reshape(semi.shape))
    return state


def run(state):
    case, semi = state["case"], state["semi"]
    if case["op"] == "rhs":
        semi.rhs_device(state["u"].data_ptr(), state["du"].data_ptr())
        return state["du"]
    semi.set_state(state["start"])
    t = semi.rk_steps(case["steps"], cfl=_CFL, t=0.0, method=case["method"])
    semi.get_state(state["out"])
    return {"u": state["out"], "t": t}


# ---- the same in plain torch, 64 bits -----------------------------------------------------------
def _saturation_pressure(T):
    c1 = (1885.0 - 4186.0) / 461.0
    c2 = (2.5e6 - (1885.0 - 4186.0) * 273.15) / 461.0
    return 610.7 * (T / 273.15) ** c1 * torch.exp(c2 * (1 / 273.15 - 1 / T))


def _half_log_ratio(x, y):
    t = (y - x) / (y + x)
    return t, torch.atanh(t)


def _ln_mean(x, y):
    t, a = _half_log_ratio(x, y)
    return 0.5 * (x + y) * torch.where(t == 0, 1.0, t / a)


def _inv_ln_mean(x, y):
    return 1 / _ln_mean(x, y)


def _stolarsky(x, y):
    d = 2 * _half_log_ratio(x, y)[1]
    ratio = torch.expm1(_GAMMA * d) / torch.expm1((_GAMMA - 1) * d)
    return x * torch.where(d == 0, 1.0, (_GAMMA - 1) / _GAMMA * ratio)


def _dot(a, b):
    return sum(p * q for p, q in zip(a, b))


class _Euler:
    """Energy or potential-temperature Euler equations with gravity, 2D or 3D: u[..., variable]."""

    def __init__(self, case):
        self.dim = 3 if case["system"].endswith("3d") else 2
        self.pt = case["system"].startswith("pt")
        self.volume, self.gravity = case.get("volume"), case.get("gravity")
        self.active = self.dim + 2

    def split(self, u):
        d = self.dim
        rho, v = u[..., 0], [u[..., 1 + k] / u[..., 0] for k in range(d)]
        if self.pt:
            p = _K * u[..., d + 1] ** _GAMMA
        else:
            p = (_GAMMA - 1) * (u[..., d + 1] - 0.5 * rho * _dot(v, v))
        return rho, v, p, u[..., d + 1], u[..., d + 2]

    def pair(self, ua, ub, n):
        ra, va, pa, ea, phia = self.split(ua)
        rb, vb, pb, eb, phib = self.split(ub)
        vna, vnb = _dot(va, n), _dot(vb, n)
        vn = 0.5 * (vna + vnb)
        if not self.pt:
            mean = _ln_mean(ra, rb)
            f1 = mean * vn
            f4 = (f1 * (0.5 * _dot(va, vb) + _inv_ln_mean(ra / pa, rb / pb) / (_GAMMA - 1))
                  + 0.5 * (pa * vnb + pb * vna))
        else:
            if self.volume == "ec":
                f1 = _ln_mean(ra, rb) * vn
                f4 = f1 * _inv_ln_mean(ra / ea, rb / eb)
            else:
                f4 = _stolarsky(ea, eb) * vn
                f1 = (_ln_mean(ra, rb) * vn if self.volume == "tec"
                      else f4 * _ln_mean(ra / ea, rb / eb))
            mean = (_ln_mean(ra, rb) if self.gravity == "waruszewski" else
                    _stolarsky(ra, rb) if self.gravity == "artiano" else 0.5 * (ra + rb))
        h = 0.5 * mean * (phib - phia)
        mom = [f1 * 0.5 * (a + b) + (0.5 * (pa + pb) + h) * k for a, b, k in zip(va, vb, n)]
        return torch.stack([f1, *mom, f4 if self.pt else f4 + h * vn], -1)

    def surface(self, ul, ur, n, c=340.0):
        rl, vl, pl, _, _ = self.split(ul)
        rr, vr, pr, _, _ = self.split(ur)
        size = torch.sqrt(_dot(n, n))
        rho, vnl, vnr = 0.5 * (rl + rr), _dot(vl, n), _dot(vr, n)
        p = 0.5 * (pl + pr) - 0.5 * c * rho * (vnr - vnl) / size
        v = 0.5 * (vnl + vnr) - (pr - pl) * size / (2 * c * rho)
        up = torch.where((v >= 0)[..., None], ul, ur)
        f = up[..., :self.active] * v[..., None]
        if not self.pt:
            f[..., -1] += torch.where(v >= 0, pl, pr) * v
        for k in range(self.dim):
            f[..., 1 + k] += p * n[k]
        return f

    def wall(self, u, n):
        size = torch.sqrt(_dot(n, n))
        e = [k / size for k in n]
        un = _dot(e, [u[..., 1 + k] for k in range(self.dim)])
        mirror = u.clone()
        for k in range(self.dim):
            mirror[..., 1 + k] -= 2 * un * e[k]
        return self.surface(u, mirror, n)

    def add_source(self, u, du):
        if self.dim == 3:
            du[..., 1] += 2 * _OMEGA * u[..., 2]
            du[..., 2] -= 2 * _OMEGA * u[..., 1]

    def speeds(self, u):
        rho, v, p, _, _ = self.split(u)
        c = torch.sqrt(_GAMMA * p / rho)
        return [w.abs() + c for w in v]

    def limit(self, u):
        return u


class _Moist:
    dim, active = 2, 6
    L, rd, rv, g = 3147620.0, 287.0, 461.0, 9.81

    def condition(self, u):
        dry = u[..., 0] - u[..., 4] - u[..., 5]
        e = u[..., 3] - 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2) / u[..., 0]
        T = (e - self.L * u[..., 4]) / (dry * 717.0 + u[..., 4] * 1424.0 + u[..., 5] * 4186.0)
        return (dry * self.rd + u[..., 4] * self.rv) * T, T, dry

    def sound(self, u, p):
        _, _, dry = self.condition(u)
        gm = ((dry * 1004.0 + u[..., 4] * 1885.0 + u[..., 5] * 4186.0)
              / (dry * 717.0 + u[..., 4] * 1424.0 + u[..., 5] * 4186.0))
        return torch.sqrt(gm * p / u[..., 0]), gm

    def pair(self, a, b, n):
        _, Ta, da = self.condition(a)
        _, Tb, db = self.condition(b)
        va = [a[..., 1 + k] / a[..., 0] for k in range(2)]
        vb = [b[..., 1 + k] / b[..., 0] for k in range(2)]
        v = [0.5 * (p + q) for p, q in zip(va, vb)]
        K = 0.25 * (_dot(va, va) + _dot(vb, vb))
        vn = _dot(v, n)
        temp = _inv_ln_mean(1 / Ta, 1 / Tb)
        p = (self.rd * 0.5 * (da + db) + self.rv * 0.5 * (a[..., 4] + b[..., 4])) / (
            0.5 * (1 / Ta + 1 / Tb))
        fd, fv, fl = (_ln_mean(q, r) * vn for q, r in
                      ((da, db), (a[..., 4], b[..., 4]), (a[..., 5], b[..., 5])))
        f1 = fd + fv + fl
        m = [f1 * v[k] + n[k] * p for k in range(2)]
        f4 = ((717.0 * temp - K) * fd + (self.L + 1424.0 * temp - K) * fv
              + (4186.0 * temp - K) * fl + _dot(v, m))
        return torch.stack([f1, *m, f4, fv, fl], -1)

    def surface(self, ul, ur, n, c=360.0):
        (pl, _, _), (pr, _, _) = self.condition(ul), self.condition(ur)
        vl = (ul[..., 1] * n[0] + ul[..., 2] * n[1]) / ul[..., 0]
        vr = (ur[..., 1] * n[0] + ur[..., 2] * n[1]) / ur[..., 0]
        size, rho = torch.sqrt(_dot(n, n)), 0.5 * (ul[..., 0] + ur[..., 0])
        p = 0.5 * (pl + pr) - 0.5 * c * rho * (vr - vl) / size
        v = 0.5 * (vl + vr) - (pr - pl) * size / (2 * c * rho)
        f = torch.where((v > 0)[..., None], ul, ur) * v[..., None]
        f[..., 3] += torch.where(v > 0, pl, pr) * v
        f[..., 1] += p * n[0]
        f[..., 2] += p * n[1]
        return f

    def wall(self, u, n):
        size = torch.sqrt(_dot(n, n))
        p, _, _ = self.condition(u)
        c, gm = self.sound(u, p)
        vn = (u[..., 1] * n[0] + u[..., 2] * n[1]) / size / u[..., 0]
        away = p * (1 + 0.5 * (gm - 1) * vn / c).clamp(min=0) ** (2 * gm / (gm - 1))
        A, B = 2 / ((gm + 1) * u[..., 0]), p * (gm - 1) / (gm + 1)
        onto = p + 0.5 * vn / A * (vn + torch.sqrt(vn * vn + 4 * A * (p + B)))
        star = torch.where(vn <= 0, away, onto)
        zero = torch.zeros_like(star)
        return torch.stack([zero, star * n[0], star * n[1], zero, zero, zero], -1)

    def add_source(self, u, du):
        p, T, dry = self.condition(u)
        du[..., 2] -= self.g * u[..., 0]
        du[..., 3] -= self.g * u[..., 2]
        vapour = 611.2 * torch.exp(17.62 * (T - 273.15) / (243.12 + T - 273.15))
        a = vapour / (self.rv * T) - u[..., 4]
        b = u[..., 0] - u[..., 4] - dry
        q = a + b - torch.sqrt(a * a + b * b)
        du[..., 4] += q
        du[..., 5] -= q

    def speeds(self, u):
        c, _ = self.sound(u, self.condition(u)[0])
        return [(u[..., 1 + k] / u[..., 0]).abs() + c for k in range(2)]

    def limit(self, u):
        return u


class _Rainy:
    dim, active = 2, 9
    cvd, cvv, cl, rd, rv, L, g = 717.0, 1424.0, 4186.0, 287.0, 461.0, 2.5e6, 9.80616

    @staticmethod
    def fall(moist, rain):
        share = (rain / (math.pi * (moist + rain) * 8.0e6)).clamp(min=0)
        return torch.where(rain > 0, 130.0 * 1.9386213994279082 * share ** 0.125, 0.0)

    @staticmethod
    def rho(u):
        return u[..., 0] + u[..., 1] + u[..., 2]

    def pair(self, a, b, n):
        va = [a[..., 3 + k] / self.rho(a) for k in range(2)]
        vb = [b[..., 3 + k] / self.rho(b) for k in range(2)]
        v = [0.5 * (p + q) for p, q in zip(va, vb)]
        K = 0.25 * (_dot(va, va) + _dot(vb, vb))
        vn = _dot(v, n)
        fall = 0.5 * n[1] * (self.fall(a[..., 6] + a[..., 7], a[..., 2])
                             + self.fall(b[..., 6] + b[..., 7], b[..., 2]))
        ia, ib = 1 / a[..., 8], 1 / b[..., 8]
        temp = _inv_ln_mean(ia, ib)

        def avg(k):
            return 0.5 * (a[..., k] + b[..., k])

        p = (self.rd * avg(0) + self.rv * avg(6)) / (0.5 * (ia + ib))
        fv, fc = _ln_mean(a[..., 6], b[..., 6]) * vn, avg(7) * vn
        fd, fr = _ln_mean(a[..., 0], b[..., 0]) * vn, avg(2) * (vn - fall)
        m = [(fd + fv + fc + fr) * v[k] + p * n[k] for k in range(2)]
        f5 = ((self.cvd * temp - K) * fd + (self.cvv * temp - K + self.L) * fv
              + (self.cl * temp - K) * (fc + fr) + _dot(v, m))
        zero = torch.zeros_like(fd)
        return torch.stack([fd, fv + fc, fr, *m, f5, zero, zero, zero], -1)

    def state(self, u):
        v = [u[..., 3 + k] / self.rho(u) for k in range(2)]
        p = (self.rd * u[..., 0] + self.rv * u[..., 6]) * u[..., 8]
        qv, ql = u[..., 6] / u[..., 0], (u[..., 7] + u[..., 2]) / u[..., 0]
        gm = 1 + (self.rd + self.rv * qv) / (self.cvd + self.cvv * qv + self.cl * ql)
        return v, p, torch.sqrt(gm * p / self.rho(u)), self.fall(u[..., 1], u[..., 2])

    def surface(self, ul, ur, n):
        def side(u):
            v, p, c, fall = self.state(u)
            vn, fn, rho = _dot(v, n), fall * n[1], self.rho(u)
            zero = torch.zeros_like(vn)
            f = torch.stack([
                u[..., 0] * vn, u[..., 1] * vn, u[..., 2] * (vn - fn),
                rho * vn * v[0] + p * n[0] - u[..., 2] * fn * v[0],
                rho * vn * v[1] + p * n[1] - u[..., 2] * fn * v[1],
                (u[..., 5] + p) * vn
                - (self.cl * u[..., 8] + 0.5 * _dot(v, v)) * u[..., 2] * fn, zero, zero, zero], -1)
            return f, vn.abs() + fn.abs(), c

        (fl, sl, cl), (fr, sr, cr) = side(ul), side(ur)
        lam = torch.maximum(sl, sr) + torch.maximum(cl, cr) * torch.sqrt(_dot(n, n))
        return 0.5 * (fl + fr) - 0.5 * lam[..., None] * (ur - ul)

    def wall(self, u, n):
        mirror = u.clone()
        mirror[..., 4] *= -1
        return self.surface(u, mirror, n)

    def add_source(self, u, du):
        T, rain = u[..., 8], u[..., 2]
        vs = _saturation_pressure(T) / (self.rv * T)
        evap = ((3.86e-3 - 9.41e-5 * (T - 273.15)) * (1 + 9.1 * rain ** 0.1875)
                * (vs - u[..., 6]) * torch.sqrt(rain))
        s = 0.001 * u[..., 7] + 1.72 * u[..., 7] * rain ** 0.875 - evap
        du[..., 1] -= s
        du[..., 2] += s
        du[..., 4] -= self.rho(u) * self.g
        du[..., 5] -= u[..., 4] * self.g

    def speeds(self, u):
        v, _, c, fall = self.state(u)
        return [v[0].abs() + c, v[1].abs() + c + fall.abs()]

    def limit(self, u):
        """The saturation equilibrium of every node, by Newton's method on its temperature:
        vapour = min(saturation density, moist density), cloud the rest, energy conserved."""
        u = u.clone()
        e = u[..., 5] - 0.5 * (u[..., 3] ** 2 + u[..., 4] ** 2) / self.rho(u)
        rain = u[..., 2].clone()
        u[..., 2] = rain.clamp(min=0)
        T, moist = u[..., 8].clone(), u[..., 1]
        for _ in range(12):
            svp = _saturation_pressure(T)
            c1 = (1885.0 - 4186.0) / 461.0
            c2 = (2.5e6 - (1885.0 - 4186.0) * 273.15) / 461.0
            dvp = svp * (c1 + c2 / T) / T
            wet = svp / (self.rv * T) < moist
            vap = torch.where(wet, svp / (self.rv * T), moist)
            slope = torch.where(wet, (dvp * T - svp) / (self.rv * T * T), 0.0)
            heat = self.cvd * u[..., 0] + self.cvv * vap + self.cl * (moist - vap + rain)
            res = heat * T + vap * self.L - e
            T = T - res / (heat + slope * ((self.cvv - self.cl) * T + self.L))
        vap = torch.minimum(_saturation_pressure(T) / (self.rv * T), moist)
        u[..., 6], u[..., 7], u[..., 8] = vap, moist - vap, T
        return u


def _lobatto(n):
    """Nodes, weights and derivative matrix on n Legendre-Gauss-Lobatto points."""
    P = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    for _ in range(3):
        inner = x[1:-1]
        x[1:-1] = inner - P.deriv()(inner) / P.deriv(2)(inner)
    w = 2 / (n * (n - 1) * P(x) ** 2)
    c = np.array([np.prod([x[i] - x[j] for j in range(n) if j != i]) for i in range(n)])
    D = np.array([[c[i] / c[j] / (x[i] - x[j]) if i != j else 0.0 for j in range(n)]
                  for i in range(n)])
    D -= np.diag(D.sum(1))
    return x, w, D


def _face_index(n, dim, elements, faces, orient):
    """Flat node index of every face node, second sides reordered by their orientation code."""
    l = torch.arange(n, device="cuda")
    if dim == 2:
        a = torch.where(orient[:, None] > 0, n - 1 - l, l)
        side, end = faces >> 1, torch.where(faces & 1 > 0, n - 1, 0)[:, None]
        i = torch.where(side[:, None] == 0, end, a)
        j = torch.where(side[:, None] == 0, a, end)
        return (elements[:, None] * n + j) * n + i
    l1, l2 = (k.reshape(1, -1) for k in torch.meshgrid(l, l, indexing="xy"))
    o = orient[:, None]
    a, b = torch.where(o & 1 > 0, l2, l1), torch.where(o & 1 > 0, l1, l2)
    a, b = torch.where(o & 2 > 0, n - 1 - a, a), torch.where(o & 4 > 0, n - 1 - b, b)
    side, end = (faces >> 1)[:, None], torch.where(faces & 1 > 0, n - 1, 0)[:, None]
    i = torch.where(side == 0, end, a)
    j = torch.where(side == 0, a, torch.where(side == 1, end, b))
    k = torch.where(side == 2, end, b)
    return ((elements[:, None] * n + k) * n + j) * n + i


class _Plain:
    """Flux-differencing DGSEM of one Cartesian system on the handle's mesh."""

    def __init__(self, case, semi):
        system = case["system"]
        self.eq = _Moist() if system == "moist2d" else _Rainy() if system == "rainy2d" else _Euler(case)
        self.n, self.dim, self.E = semi.n, self.eq.dim, semi.nelements
        self.members = case.get("members", 1)
        _, w, D = _lobatto(self.n)
        S = 2 * D
        S[0, 0] += 1 / w[0]
        S[-1, -1] -= 1 / w[-1]
        self.S, self.w = _dev(S), float(w[0])
        self.ja = _dev(semi.contravariant_vectors).reshape(-1, self.dim, self.dim)
        self.ij = _dev(semi.inverse_jacobian).reshape(-1)
        ie, ifc, fl, be, bf, _ = (_dev(np.asarray(a, dtype=np.int64))
                                  for a in semi._H.connectivity_arrays)
        none = torch.zeros_like(ie[:, 0])
        self.left = _face_index(self.n, self.dim, ie[:, 0], ifc[:, 0], none)
        self.right = _face_index(self.n, self.dim, ie[:, 1], ifc[:, 1], fl)
        self.edge = _face_index(self.n, self.dim, be, bf, torch.zeros_like(be))
        self.fl, self.fb = ifc[:, 0], bf

    def normal(self, q, faces):
        d, sign = faces >> 1, torch.where(faces & 1 > 0, 1.0, -1.0)
        ja = self.ja[q, d[:, None].expand_as(q)]
        return [ja[..., k] * sign[:, None] for k in range(self.dim)]

    def rhs(self, u):
        shape, n, dim, eq = u.shape, self.n, self.dim, self.eq
        flat = u.reshape(-1, shape[-1])
        acc = torch.zeros(flat.shape[0], eq.active, dtype=u.dtype, device=u.device)
        grid = (n,) * dim
        step = max(1, 40_000_000 // (n ** (dim + 1) * 40))
        for e in range(0, self.E, step):
            cut = slice(e * n ** dim, min(self.E, e + step) * n ** dim)
            for d in range(dim):
                def lines(a):
                    return a.reshape(-1, *grid, a.shape[-1]).movedim(dim - d, -2)
                v, ja = lines(flat[cut]), lines(self.ja[cut, d])
                nrm = 0.5 * (ja[..., :, None, :] + ja[..., None, :, :])
                F = eq.pair(v[..., :, None, :], v[..., None, :, :],
                            [nrm[..., k] for k in range(dim)])
                part = torch.einsum("ab,...abv->...av", self.S, F)
                acc[cut] += part.movedim(-2, dim - d).reshape(-1, eq.active)
        F = eq.surface(flat[self.left], flat[self.right], self.normal(self.left, self.fl)) / self.w
        B = eq.wall(flat[self.edge], self.normal(self.edge, self.fb)) / self.w
        for q, f in ((self.left, F), (self.right, -F), (self.edge, B)):
            acc.index_add_(0, q.reshape(-1), f.reshape(-1, eq.active))
        du = torch.zeros_like(flat)
        du[:, :eq.active] = -acc * self.ij[:, None]
        eq.add_source(flat, du)
        return du.reshape(shape)

    def time_step(self, u):
        flat = u.reshape(-1, u.shape[-1])
        lam = self.eq.speeds(flat)
        top = sum((sum(self.ja[:, d, k] * lam[k] for k in range(self.dim)).abs() * self.ij.abs())
                  .reshape(self.E, -1).amax(1) for d in range(self.dim))
        return _CFL * 2 / (self.n * top.reshape(self.members, -1).amax(1))

    def limit(self, u):
        return self.eq.limit(u)

    def spread(self, dt):
        per = self.E // self.members
        return dt.repeat_interleave(per).reshape(-1, *(1,) * (self.dim + 1))


class _PlainSwe:
    """Covariant shallow water of one member: weak form with Lax-Friedrichs fluxes, or the split
    entropy-conserving form; state [elements, n, n, 3], metric terms as the mesh gives them."""

    def __init__(self, case, semi, m):
        aux = _dev(np.asarray(semi._H.aux[m]))
        mesh = getattr(semi, "meshes", [getattr(semi, "mesh", None)])[m]
        self.n, self.ec = semi._H.ns[m], case["form"] == "ec"
        basis = getattr(semi, "solvers", [getattr(semi, "solver", None)])[m].basis
        ie, ifc, fl, _, _ = (_dev(np.asarray(a, dtype=np.int64))
                             for a in mesh.connectivity(basis).arrays())
        _, w, D = _lobatto(self.n)
        S = 2 * D
        S[0, 0] += 1 / w[0]
        S[-1, -1] -= 1 / w[-1]
        self.S, self.w = _dev(S), float(w[0])
        self.weak = _dev(-(D.T * w[None, :]) / w[:, None])
        self.aux = aux.reshape(-1, self.n, self.n, 26)
        x = _dev(np.asarray(semi._H.xyz[m])).reshape(self.aux.shape[:3] + (3,))
        self.f = 2 * _OMEGA * x[..., 2] / x.norm(dim=-1)
        none = torch.zeros_like(fl)
        self.left = _face_index(self.n, 2, ie[:, 0], ifc[:, 0], none)
        self.right = _face_index(self.n, 2, ie[:, 1], ifc[:, 1], fl)
        self.fl, self.fr = ifc[:, 0], ifc[:, 1]
        self.members = 1

    @staticmethod
    def gcon(a):
        return [[a[..., 16], a[..., 17]], [a[..., 17], a[..., 18]]]

    def flux(self, u, a, o):
        J, G = a[..., 12], self.gcon(a)
        f = [J * u[..., 1 + o]]
        for c in range(2):
            t = u[..., 1 + c] * u[..., 1 + o] / u[..., 0]
            f.append(J * (t if self.ec else t + G[c][o] * 0.5 * _GRAVITY * u[..., 0] ** 2))
        return torch.stack(f, -1)

    def pair_ec(self, ua, ub, aa, ab, o):
        Ja, Jb = aa[..., 12], ab[..., 12]
        va = [ua[..., 1 + c] / ua[..., 0] for c in range(2)]
        vb = [ub[..., 1 + c] / ub[..., 0] for c in range(2)]
        m = 0.5 * (Ja * ua[..., 1 + o] + Jb * ub[..., 1 + o])
        G = self.gcon(aa)
        cov = [ab[..., 13] * vb[0] + ab[..., 14] * vb[1], ab[..., 14] * vb[0] + ab[..., 15] * vb[1]]
        ph = _GRAVITY * ua[..., 0] * (ub[..., 0] + ab[..., 19] - aa[..., 19])
        F = [m]
        N = [torch.zeros_like(m)]
        for c in range(2):
            F.append(m * 0.5 * (va[c] + vb[c]))
            N.append(0.5 * Ja * (0.5 * ua[..., 1 + o] * (G[c][0] * cov[0] + G[c][1] * cov[1] - vb[c])
                                 + G[c][o] * ph))
        return torch.stack(F, -1), torch.stack(N, -1)

    def side(self, mine, other, am, ao, faces):
        """Outward flux of one side, the neighbour's velocity taken through global coordinates."""
        glob = [ao[..., r] * other[..., 1] + ao[..., 3 + r] * other[..., 2] for r in range(3)]
        there = torch.stack([other[..., 0]] + [
            sum(am[..., 6 + r + 2 * k] * glob[k] for k in range(3)) for r in range(2)], -1)
        plus = (faces & 1 > 0)[:, None, None]
        L, R = torch.where(plus, mine, there), torch.where(plus, there, mine)
        out = []
        for o in range(2):
            J, G = am[..., 12], self.gcon(am)
            if self.ec:
                m = 0.5 * J * (L[..., 1 + o] + R[..., 1 + o])
                F = torch.stack([m] + [m * 0.5 * (L[..., 1 + c] / L[..., 0] + R[..., 1 + c] / R[..., 0])
                                       for c in range(2)], -1)
            else:
                F = 0.5 * (self.flux(L, am, o) + self.flux(R, am, o))

            def speed(u):
                return (u[..., 1 + o] / u[..., 0]).abs() + torch.sqrt(G[o][o] * u[..., 0] * _GRAVITY)

            F = F - (0.5 * J * torch.maximum(speed(L), speed(R)))[..., None] * (R - L)
            if self.ec:
                ph = 0.5 * J * _GRAVITY * L[..., 0] * R[..., 0]
                F = F + torch.stack([torch.zeros_like(ph), G[0][o] * ph, G[1][o] * ph], -1)
            out.append(F)
        F = torch.where((faces >> 1 == 0)[:, None, None], out[0], out[1])
        return torch.where(plus, F, -F)

    def rhs(self, u):
        aux, n = self.aux, self.n
        acc = torch.zeros_like(u)
        for o, axis in ((0, 2), (1, 1)):
            v, a = u.movedim(axis, -2), aux.movedim(axis, -2)
            if self.ec:
                F, N = self.pair_ec(v[..., :, None, :], v[..., None, :, :], a[..., :, None, :],
                                    a[..., None, :, :], o)
                off = self.S * (1 - torch.eye(n, device="cuda", dtype=u.dtype))
                part = (torch.einsum("ab,...abv->...av", off, F)
                        + torch.einsum("ab,...abv->...av", self.S, N))
            else:
                part = torch.einsum("ab,...bv->...av", self.weak, self.flux(v, a, o))
            acc += part.movedim(-2, axis)
        flat, fa = u.reshape(-1, 3), aux.reshape(-1, 26)
        out = acc.reshape(-1, 3)
        for q, r, faces in ((self.left, self.right, self.fl), (self.right, self.left, self.fr)):
            F = self.side(flat[q], flat[r], fa[q], fa[r], faces) / self.w
            out.index_add_(0, q.reshape(-1), F.reshape(-1, 3))
        return -out.reshape(u.shape) / aux[..., 12:13] + self.source(u)

    def source(self, u):
        a = self.aux
        C = [[[a[..., 20], a[..., 21]], [a[..., 21], a[..., 22]]],
             [[a[..., 23], a[..., 24]], [a[..., 24], a[..., 25]]]]
        G = self.gcon(a)
        g = [[a[..., 13], a[..., 14]], [a[..., 14], a[..., 15]]]
        T = [[u[..., 1 + r] * u[..., 1 + c] / u[..., 0] for c in range(2)] for r in range(2)]
        pressure = 0 if self.ec else 0.5 * _GRAVITY * u[..., 0] ** 2
        two = range(2)
        s = [sum(C[k][r][c] * (T[r][c] + pressure * G[r][c]) for r in two for c in two) for k in two]
        if self.ec:
            cov = [[sum(g[r][k] * T[k][c] for k in two) for c in two] for r in two]
            w = [sum(C[k][i][c] * cov[k][c] for k in two for c in two) for i in two]
            s = [0.5 * (s[k] - sum(G[k][i] * w[i] for i in two)) for k in two]
        fJ = self.f * a[..., 12]
        return torch.stack([torch.zeros_like(fJ)] + [
            -(s[k] + fJ * (G[k][1] * u[..., 1] - G[k][0] * u[..., 2])) for k in two], -1)

    def time_step(self, u):
        top = sum(((u[..., 1 + o] / u[..., 0]).abs()
                   + torch.sqrt(self.gcon(self.aux)[o][o] * u[..., 0] * _GRAVITY))
                  .reshape(u.shape[0], -1).amax(1) for o in range(2))
        return _CFL * 2 / (self.n * top.amax(0, keepdim=True))

    def limit(self, u):
        return u

    def spread(self, dt):
        return dt.reshape(1, 1, 1, 1)


def _integrate(plain, u, steps, method):
    """Steps of one of the three schemes at dt = cfl * max_dt; returns the state and the times."""
    A = [0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238,
         -3550918686646 / 2091501179385, -1275806237668 / 842570457699]
    B = [1432997174477 / 9575080441755, 5161836677717 / 13612068292357,
         1720146321549 / 2090206949498, 3134564353537 / 4481467310338,
         2277821191437 / 14882151754819]
    t = torch.zeros(plain.members, dtype=u.dtype, device=u.device)
    for _ in range(steps):
        dt = plain.time_step(u)
        t += dt
        h = plain.spread(dt)
        if method == "CarpenterKennedy2N54":
            k = torch.zeros_like(u)
            for a, b in zip(A, B):
                k = a * k + h * plain.rhs(u)
                u = plain.limit(u + b * k)
        elif method == "SSPRK43":
            start = u
            for s in range(4):
                u = u + 0.5 * h * plain.rhs(u)
                u = 2 / 3 * start + 1 / 3 * u if s == 2 else u
        else:
            start = u
            u = u + h * plain.rhs(u)
            u = 0.75 * start + 0.25 * (u + h * plain.rhs(u))
            u = 1 / 3 * start + 2 / 3 * (u + h * plain.rhs(u))
    return u, t


def exact(case, seed):
    semi = _semi(case)
    u = _initial_state(case, semi, seed)
    if case["system"] == "swe":
        parts, times, at = [], [], 0
        for m in range(case["members"]):
            plain = _PlainSwe(case, semi, m)
            count = plain.aux[..., 0].numel() * 3
            um = u.reshape(-1)[at:at + count].reshape(plain.aux.shape[:3] + (3,))
            at += count
            um, t = _integrate(plain, um, case["steps"], case["method"])
            parts.append(um.reshape(-1))
            times.append(float(t[0]))
        out = torch.cat(parts).cpu().numpy().reshape(semi.shape)
        return {"u": out, "t": times[0] if len(times) == 1 else np.array(times)}
    plain = _Plain(case, semi)
    if case["op"] == "rhs":
        return plain.rhs(u)
    u, t = _integrate(plain, u, case["steps"], case["method"])
    t = t.cpu().numpy()
    return {"u": u.cpu().numpy().reshape(semi.shape), "t": float(t[0]) if t.size == 1 else t}
