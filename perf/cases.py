"""Performance cases of the MLS-MPM step: what a program built on this library calls, and how often.

Every case is one call (or one call and the read-back that follows it) on a scene that is already on
the device, in the middle of its motion: the blocks move, spin and are strained, plastic strain and
temperature are not at their initial values, positions are jittered and blocks sit anywhere relative
to the cells. Kinds:

  frame    MPM3.frame, the interactive loop of the reference's worker: the caller's FP64 arrays go in
           and come back every displayed frame, and the viewer's FP32 buffers are filled from them
  run      Solver.run over several requested steps, then the whole state into the caller's FP32 arrays
  soil     the same for snow, sand, cohesive soil and foam in one scene (history laws)
  regular  the same with the reference's default position regularisation after every substep
  batch    Batch.run, a V&V ensemble of scenes of uneven size, then the state
  heat     Solver.exchange_heat, the particle-pair heat exchange of one frame, then the temperatures
  plane    SolidMPM.frame, one frame of the 2D class

Sizes are those of the repository's scenes and tests, their halves and doubles, and odd ones.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "summer-particle-lab_b200"))
from mpm_b200 import _lib, params, scenes, solid_mpm  # noqa: E402
from mpm_b200.mpm3 import MPM3, Sim3  # noqa: E402
from mpm_b200.solver import Batch, Solver  # noqa: E402

SOIL = (2, 3, 8, 9)  # snow, sand, cohesive Drucker-Prager, foam


def listed():
    return [
        # the elastic cube of the tests (13,824 particles) shown at 60 frames a second: the smallest
        # 3D call, bound by launches and copies
        {"name": "frame_cube", "kind": "frame", "bx": 12, "by": 12, "bz": 12, "grid": 32, "model": 0, "newton": 0},
        # one 2D frame of a panel near the 2D class's particle capacity
        {"name": "plane_panel", "kind": "plane", "width": 301.0, "height": 303.0, "gravity": "center"},
        # a small metal part, one requested step per call: a host loop that looks at every step
        {"name": "step_part", "kind": "run", "bx": 19, "by": 13, "bz": 23, "grid": 48, "model": 5, "newton": 0,
         "conduct": 0, "steps": 1},
        # an eighth of the 2M drop (the sub-block the CPU baseline uses), several steps per call
        {"name": "j2_262144", "kind": "run", "bx": 64, "by": 16, "bz": 32, "grid": 128, "model": 5, "newton": 0,
         "conduct": 0, "steps": 10},
        # the headline scene: 2,097,152 particles, J2 with linear hardening, 128^3 grid
        {"name": "j2_2097152", "kind": "run", "bx": 64, "by": 64, "bz": 64, "grid": 128, "model": 5, "newton": 0,
         "conduct": 0, "steps": 16},
        # the largest single scene: thermal softening and plastic heating, 4,096,000 particles, 160^3 grid
        {"name": "thermal_4096000", "kind": "run", "bx": 80, "by": 80, "bz": 80, "grid": 160, "model": 10, "newton": 0,
         "conduct": 0, "steps": 10},
        # Johnson-Cook impact, ragged block, the reference's bisection return
        {"name": "johnson_cook", "kind": "run", "bx": 53, "by": 37, "bz": 61, "grid": 96, "model": 7, "newton": 0,
         "conduct": 0, "steps": 8},
        # the coupled scene at half its resolution: thermal J2 with grid heat conduction
        {"name": "conducting", "kind": "run", "bx": 64, "by": 64, "bz": 32, "grid": 128, "model": 10, "newton": 0,
         "conduct": 1, "steps": 8},
        # snow, sand, soil and foam layers in one scene: history laws on the eigen path, four materials
        {"name": "soil_layers", "kind": "soil", "bx": 34, "by": 21, "bz": 30, "grid": 64, "steps": 1},
        # an elastic body with the reference's default regularisation after every substep
        {"name": "regular_body", "kind": "regular", "bx": 32, "by": 30, "bz": 33, "grid": 64, "model": 0, "steps": 1},
        # an ensemble of 48 scenes, 5,832 to 195,112 particles each, 64 substeps of their own dt
        {"name": "ensemble_48", "kind": "batch", "scenes": 48, "side_lo": 9, "side_hi": 29, "steps": 64},
        # heat exchange of a two-material body, pairs closer than the reference's radius to spacing ratio
        {"name": "heat_pairs", "kind": "heat", "bx": 40, "by": 36, "bz": 31, "grid": 64},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def block(lo, hi, side):
        """A block of about lo..hi particles (log-uniform) with unequal odd or even sides below `side` cells."""
        cells = log(lo, hi) / 8
        a, b = rng.uniform(.7, 1.4), rng.uniform(.7, 1.4)
        e = cells ** (1 / 3)
        c = [max(3, int(round(s))) for s in (e * a, e * b, e / (a * b))]
        return [min(side, v) for v in c]

    kind = rng.choice(["run", "run", "run", "frame", "soil", "regular", "batch", "heat", "plane"])
    if kind == "plane":
        return {"kind": kind, "width": round(log(60, 420), 1), "height": round(log(60, 420), 1),
                "gravity": rng.choice(["center", "none"])}
    if kind == "batch":
        lo = rng.randrange(8, 14)
        return {"kind": kind, "scenes": rng.randrange(3, 48), "side_lo": lo, "side_hi": rng.randrange(lo + 2, 29),
                "steps": rng.choice([20, 64, 100])}
    if kind == "frame":
        b = block(3e3, 6e4, 26)
        return {"kind": kind, "bx": b[0], "by": b[1], "bz": b[2], "grid": rng.choice([32, 40]),
                "model": rng.choice([0, 1]), "newton": 0}
    if kind in ("soil", "heat", "regular"):
        b = block(1e4, 3e5, 48)
        c = {"kind": kind, "bx": b[0], "by": b[1], "bz": b[2], "grid": 64}
        if kind != "heat":
            c["steps"] = 1
        if kind == "regular":
            c["model"] = rng.choice([0, 1])
        return c
    model = rng.choice([0, 4, 5, 6, 7, 10])
    grid = rng.choice([64, 96, 128, 160])
    b = block(1e4, 3e6, grid // 2)
    return {"kind": kind, "bx": b[0], "by": b[1], "bz": b[2], "grid": grid, "model": model,
            "newton": int(model in (6, 7) and rng.random() < .5), "conduct": int(model == 10 and rng.random() < .5),
            "steps": rng.choice([1, 4, 8])}


# ---- inputs -----------------------------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _material(case, model, k=0):
    """The repository's materials: soft elastic cube, aluminium, its thermal and Johnson-Cook forms, soils."""
    if case["kind"] == "soil":
        return params.Material.reference_units(model, E=1e6, density=1000.0)
    if case["kind"] == "heat":
        cp, cond = ((4180.0, 0.6), (450.0, 80.0))[k]
        return params.Material(model=0, mu=4e4, lam=4e4, density=(1000.0, 7870.0)[k], specific_heat=cp, conductivity=cond)
    if model in (0, 1):
        return params.Material.from_young(model, 1e5, .3, density=1000.0)
    if model in (6, 7):
        return scenes.johnson_cook_metal(model)
    if model == 10:
        hot = 293.0 + .999 * 250e6 / .3e6
        return scenes.aluminium_j2(model, T_ref=293.0, T_hot=hot, hot_ratio=.001, heat_fraction=.9, specific_heat=900.0)
    return scenes.aluminium_j2(model)


def _soft(case):
    return case["kind"] in ("soil", "heat") or case["model"] in (0, 1)


def _dt(case):
    """Requested time step: a 60 Hz frame (interactive), 1 / 240 s (soft bodies), 2e-6 s (metal)."""
    return 1 / 60 if case["kind"] in ("frame", "heat") else 1 / 240 if _soft(case) else 2e-6


def _inputs(case, seed):
    """Particle state of a block in motion, FP64 on the GPU (a dict of tensors)."""
    dev = _dev()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    rnd = lambda *s: torch.rand(*s, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
    grid = case["grid"]
    h = 1.0 / grid
    b = [case["bx"], case["by"], case["bz"]]
    drift = rnd(3).cpu().tolist()
    lo = [(grid - b[0]) // 2 + drift[0], 1 + .5 * drift[1], (grid - b[2]) // 2 + drift[2]]
    if not _soft(case):
        lo[1] += 1 + grid // 16
    ax = [torch.arange(2 * n, device=dev, dtype=torch.float64) * .5 + .25 for n in b]
    x = torch.stack(torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")[::-1], -1).reshape(-1, 3)
    n = x.shape[0]
    x = (x + .25 * (2 * rnd(n, 3) - 1) + torch.tensor(lo, device=dev, dtype=torch.float64)) * h
    V = torch.full((n,), h ** 3 / 8, device=dev, dtype=torch.float64)
    # velocity: a mean, a spin and a standing wave; C is its gradient
    size = h * max(b)
    speed = {"frame": 1.0, "regular": .5, "soil": 1.0, "heat": 0.0}.get(case["kind"], 1.0 if _soft(case) else 20.0)
    r = (x - x.mean(0)) / size
    A = speed * (2 * rnd(3, 3) - 1)
    ph = 2 * math.pi * rnd(3)
    k = math.pi * (1 + rnd(3))
    v = r @ A.T + speed * .5 * torch.sin(r[:, [1, 2, 0]] * k + ph)
    v[:, 1] -= .5 * speed
    C = (A / size).expand(n, 3, 3).clone()
    for a in range(3):
        C[:, a, (a + 1) % 3] += speed * .5 * k[a] / size * torch.cos(r[:, (a + 1) % 3] * k[a] + ph[a])
    strain = 5e-3 if _soft(case) else 1.5e-3
    S = 2 * rnd(3, 3) - 1
    F = torch.eye(3, device=dev, dtype=torch.float64) + strain * (
        S * (.5 + .5 * torch.sin(2 * math.pi * r[:, 0] + ph[0]))[:, None, None])
    i = dict(x=x, v=v, C=C, F=F, V=V, T=293.0 + 200.0 * rnd(n), ep=.02 * rnd(n),
             mat=torch.zeros(n, dtype=torch.int64, device=dev))
    if case["kind"] == "soil":
        i["mat"] = torch.clamp((4 * (x[:, 1] - x[:, 1].min()) / (h * b[1])).long(), 0, 3)
        i["T"] = None
    if case["kind"] == "heat":
        i["mat"] = (r[:, 0] + .2 * torch.sin(9 * r[:, 1]) > 0).long()
        i["T"] = 20.0 + 280.0 * (torch.sin(7 * r[:, 2] + ph[0]) > 0) + 10 * rnd(n)
        i["ep"] = None
    elif case["kind"] != "soil":
        if case["model"] in (0, 1):
            i["ep"] = None
        if case["model"] not in (6, 10):
            i["T"] = None
    return i


def _materials(case):
    if case["kind"] == "soil":
        return [_material(case, m) for m in SOIL]
    if case["kind"] == "heat":
        return [_material(case, 0, k) for k in (0, 1)]
    return [_material(case, case["model"])]


def _domain(case):
    return params.Domain(lower=(0, 0, 0), upper=(1, 1, 1), H=1.0 / case["grid"], gravity=(0, -9.8, 0), sticky_floor=True)


def _mass(i, mats):
    rho = torch.tensor([m.density for m in mats], dtype=torch.float64, device=i["V"].device)
    return i["V"] * rho[i["mat"]]


def _scene(case, seed):
    i, mats = _inputs(case, seed), _materials(case)
    f = lambda a: None if a is None else a.cpu().numpy()  # noqa: E731
    n = i["x"].shape[0]
    return scenes.Scene(name="case", domain=_domain(case), materials=mats, x=f(i["x"]), v=f(i["v"]),
                        m=f(_mass(i, mats)), V=f(i["V"]), mat=f(i["mat"]).astype(np.int32), T=f(i["T"]),
                        F=f(i["F"]).reshape(n, 9), C=f(i["C"]).reshape(n, 9), ep=f(i["ep"]))


def _batch_cases(case):
    """Scene k of an ensemble: sides between side_lo and side_hi, grids from 32 to 96 cells, ideal and hardening J2."""
    out = []
    for k in range(case["scenes"]):
        t = k / max(1, case["scenes"] - 1)
        side = int(round(case["side_lo"] + (case["side_hi"] - case["side_lo"]) * t * t))
        out.append({"kind": "run", "bx": side, "by": side, "bz": side, "grid": max(32 + (k * 37) % 65, 2 * side),
                    "model": 4 + k % 2, "newton": 0, "conduct": 0, "steps": case["steps"]})
    return out


class Readback:
    """The caller's FP32 arrays in pinned memory, filled by mpm_download_particles."""

    def __init__(self, sol, fields):
        self.sol, self.n = sol, sol.n
        pin = lambda *s: torch.empty(*s, dtype=torch.float32, pin_memory=True)  # noqa: E731
        self.out, p = {}, _lib.MpmParticles(dtype=_lib.F32)
        for f in fields:
            names = {"x": ("x", "y", "z"), "v": ("vx", "vy", "vz"), "F": ("F",), "C": ("C",), "ep": ("plastic",),
                     "T": ("temperature",), "jp": ("jp",), "dilation": ("dilation",), "enthalpy": ("enthalpy",)}[f]
            for name in names:
                self.out[name] = pin(self.n, 9) if f in "FC" else pin(self.n)
                setattr(p, name, ctypes.c_void_p(self.out[name].data_ptr()))
        self.p = p

    def __call__(self):
        self.sol._check(_lib.lib().mpm_download_particles(self.sol.h, ctypes.byref(self.p)))
        return self.out


def _fields(case):
    if case["kind"] == "heat":
        return ("T", "enthalpy")
    if case["kind"] == "soil":
        return ("x", "v", "F", "C", "ep", "jp", "dilation")
    f = ["x", "v", "F", "C"]
    if case["kind"] == "batch" or case["model"] >= 2:
        f.append("ep")
    if case["kind"] != "batch" and case["model"] in (6, 10):
        f.append("T")
    return tuple(f)


def _reg(case):
    h = 1.0 / case["grid"]
    return dict(spacing=.6 * h, volume_unit=h ** 3 / 8, max_speed=2.0, rate=40.0)


def _heat(case):
    """Radius 8 at spacing 2.8, the reference's ratio, for particles half a cell apart."""
    h = 1.0 / case["grid"]
    return dict(radius=.5 * h * 8 / 2.8, geometry=.05 * h, heat_rate=20.0)


def _plane_inputs(case, seed):
    s = solid_mpm.SolidSim(scene="empty", gravity=case["gravity"])
    w, h = case["width"], case["height"]
    solid_mpm.create_body(s, -w / 2, -h / 2, w / 2, h / 2)
    g = np.random.default_rng(int(seed))
    n = s.count
    x, y = s.x[:n].copy(), s.y[:n].copy()
    a, b, c = g.uniform(-1, 1, 3)
    s.x[:n] += g.uniform(-.4, .4, n)
    s.y[:n] += g.uniform(-.4, .4, n)
    s.vx[:n] = 30 * a + 20 * np.sin(y / h * 3 + b) + g.uniform(-2, 2, n)
    s.vy[:n] = 30 * c + 20 * np.sin(x / w * 3 + a) + g.uniform(-2, 2, n)
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plane":
        s = _plane_inputs(case, seed)
        s.mpm = solid_mpm.SolidMPM(s.capacity)
        return {"kind": kind, "sim": s}
    if kind == "frame":
        sc = _scene(case, seed)
        s = Sim3(sc.n)
        s.count = sc.n
        for k in range(3):
            (s.x, s.y, s.z)[k][:] = sc.x[:, k]
            (s.vx, s.vy, s.vz)[k][:] = sc.v[:, k]
        s.mass[:], s.volume[:] = sc.m, sc.V
        return {"kind": kind, "sim": s, "mpm": MPM3(sc.n, sc.domain, {0: sc.materials[0]}), "dt": _dt(case)}
    if kind == "batch":
        sub = [_scene(c, seed * 1000 + k) for k, c in enumerate(_batch_cases(case))]
        for sc in sub:
            sc.T = None
        sol = Batch(sub)
        sol.upload()
        sol.scenes = [sc.domain for sc in sub]  # the host arrays are not needed any more
        return {"kind": kind, "sol": sol, "steps": case["steps"], "read": Readback(sol, _fields(case))}
    sc = _scene(case, seed)
    sol = Solver(sc.domain, sc.n)
    sol.upload(sc)
    if kind == "run" and case["conduct"]:
        sol.set_conduction(150.0, 2700.0, 900.0)
    if kind == "run" and case["newton"]:
        sol.set_return_mode(mode="newton")
    if kind == "regular":
        sol.set_regularizer(True, **_reg(case))
    s = {"kind": kind, "sol": sol, "dt": _dt(case), "read": Readback(sol, _fields(case))}
    if kind == "heat":
        s["heat"] = _heat(case)
    else:
        s["steps"] = case["steps"]
    return s


def run(state):
    kind = state["kind"]
    if kind == "plane":
        s = state["sim"]
        s.mpm.frame(s)
        return [a[:s.count] for a in (s.x, s.y, s.vx, s.vy)]
    if kind == "frame":
        s = state["sim"]
        state["mpm"].frame(s, state["dt"])
        return [a[:s.count].astype(np.float32) for a in (s.x, s.y, s.z, s.vx, s.vy, s.vz)]
    if kind == "batch":
        state["sol"].run(state["steps"])
    elif kind == "heat":
        state["sol"].exchange_heat(state["dt"], **state["heat"])
    else:
        state["sol"].run(state["dt"], state["steps"])
    return state["read"]()


# ---- the work of a pass -----------------------------------------------------------------------------

def _particles(case):
    return 8 * case["bx"] * case["by"] * case["bz"]


def _substeps(case):
    m = _materials(case)[0]
    cfl = .4 / case["grid"] / m.wave_speed
    return case.get("steps", 1) * math.ceil(_dt(case) / cfl)


def work(case):
    """Every substep streams the particle state once: position and F in and out, mass and volume in, and
    each law's scalars in and out; the call's inputs and outputs cross once. Per particle and
    substep the two transfers take 27 nodes x (22 + 12) multiply-adds and the law some 300 operations."""
    kind = case["kind"]
    if kind == "plane":
        n = (math.floor(case["width"] / 3.6) + 1) * (math.floor(case["height"] / 3.6) + 1)
        return {"bytes": n * (8 * 64 + 42), "flops": n * 8 * 500}
    if kind == "batch":
        c = _batch_cases(case)
        n = sum(_particles(s) for s in c)
        return {"bytes": n * (case["steps"] * 112 + 100), "flops": n * case["steps"] * 2100}
    n = _particles(case)
    if kind == "heat":
        return {"bytes": n * (16 + 8 + 8), "flops": n * 98 * 2 * 20}
    sub = _substeps(case)
    if kind == "frame":
        return {"bytes": n * (sub * 104 + 96), "flops": n * sub * 2100}
    scalars = sum({"ep": 8, "T": 8, "jp": 8}.get(f, 0) for f in _fields(case))
    back = 4 * sum({"x": 3, "v": 3, "F": 9, "C": 9}.get(f, 1) for f in _fields(case))
    flops = 2100 + (400 if kind in ("soil", "regular") else 0)
    return {"bytes": n * (sub * (104 + scalars) + back), "flops": n * sub * flops}


# ---- the same in 64 bits ----------------------------------------------------------------------------

def _eig(B):
    """Eigen-decomposition of many symmetric 3x3 matrices, in pieces the solver takes."""
    parts = [torch.linalg.eigh(p) for p in B.split(16384)]
    return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])


def _diag(U, d):
    return (U * d[:, None, :]) @ U.transpose(1, 2)


def _flow(m, ep, rate, T):
    f = (m.yield_stress + m.hardening * torch.clamp(ep, min=0) ** m.jc_n) * (
        1 + m.jc_C * torch.log(torch.clamp(rate / m.jc_rate0, min=1)))
    if m.model == 6:
        f = f * (1 - torch.clamp((T - m.T_ref) / (m.T_melt - m.T_ref), 0, 1) ** m.jc_m)
    return f


def _law(m, s, do_return, dt):
    """Kirchhoff stress of the state (and the J2-type return before it): updates F, ep and T in s."""
    F = s["F"]
    eye = torch.eye(3, device=F.device, dtype=F.dtype)
    if m.model == 1:
        J = torch.linalg.det(F)[:, None, None]
        return m.mu * (F @ F.transpose(1, 2) - eye) + m.lam * torch.log(J) * eye
    lam, U = _eig(F @ F.transpose(1, 2))
    if m.model == 0:
        J = torch.linalg.det(F)
        sg = torch.sqrt(lam)
        return _diag(U, 2 * m.mu * (sg * sg - sg) + (m.lam * (J - 1) * J)[:, None])
    e = .5 * torch.log(lam)
    tr = e.sum(1)
    dev = e - tr[:, None] / 3
    ln = dev.norm(dim=1)
    scale = torch.ones_like(ln)
    if do_return:
        J, ep = torch.exp(tr), s["ep"]
        q, slope = math.sqrt(6) * m.mu * ln / J, 3 * m.mu / J
        if m.model in (6, 7):
            lo, hi = torch.zeros_like(q), q / slope
            for _ in range(60):
                mid = .5 * (lo + hi)
                up = q - slope * mid > _flow(m, ep + mid, mid / dt, s["T"])
                lo, hi = torch.where(up, mid, lo), torch.where(up, hi, mid)
            dep = torch.where(q > _flow(m, ep, 0 * q, s["T"]), .5 * (lo + hi), 0 * q)
        else:
            soft = torch.ones_like(q)
            if m.model == 10:
                soft = 1 - (1 - m.hot_ratio) * torch.clamp((s["T"] - m.T_ref) / (m.T_hot - m.T_ref), 0, 1)
            H = 0.0 if m.model == 4 else m.hardening
            dep = torch.clamp(q - (m.yield_stress + H * ep) * soft, min=0) / (slope + H * soft)
        scale = torch.where(dep > 0, torch.clamp(1 - math.sqrt(1.5) * dep / torch.clamp(ln, min=1e-20), min=0), scale)
        s["F"] = _diag(U, torch.exp((scale - 1)[:, None] * dev)) @ F
        s["ep"] = ep + dep
        if s["T"] is not None:
            s["T"] = s["T"] + m.heat_fraction / m.specific_heat * math.sqrt(6) * m.mu * scale * ln * dep * s["V"] / s["m"]
    return _diag(U, 2 * m.mu * (tr[:, None] / 3 + scale[:, None] * dev) + (m.lam * tr)[:, None])


class _Exact:
    def __init__(self, case, seed):
        self.d, self.mat = _domain(case), _materials(case)[0]
        s = _inputs(case, seed)
        if case["kind"] == "frame":
            s["F"] = torch.eye(3, device=s["F"].device, dtype=torch.float64).expand_as(s["F"]).clone()
            s["C"] = torch.zeros_like(s["C"])
        s["m"] = _mass(s, [self.mat])
        self.s, self.h = s, 1.0 / case["grid"]
        self.n = case["grid"] + 5
        self.o = -2 * self.h
        self.tau = _law(self.mat, s, False, 0.0)

    def stable(self):
        s, m = self.s, self.mat
        a = s["F"].abs()
        st = torch.clamp(a.sum(2).amax(1) * a.sum(1).amax(1), min=1)
        if m.model == 1:
            st = torch.maximum(st, 1 / torch.clamp(torch.linalg.det(s["F"]), min=.05))
        c = torch.sqrt((m.lam + 2 * m.mu) * s["V"] / s["m"])
        wave = max(1.0, float((s["v"].norm(dim=1) + c * st).max()))
        grad = max(1.0, float(s["C"].abs().sum((1, 2)).max()))
        return min(self.d.cfl * self.h / wave, self.d.grad_limit / grad)

    def substep(self, dt):
        s, h, n = self.s, self.h, self.n
        q = (s["x"] - self.o) / h
        base = torch.clamp(torch.floor(q - .5).long(), 0, n - 3)
        t = q - base
        w = torch.stack([.5 * (1.5 - t) ** 2, .75 - (t - 1) ** 2, .5 * (t - .5) ** 2], 1)
        off = [(i, j, k) for k in range(3) for j in range(3) for i in range(3)]
        flat = (base[:, 2] * n + base[:, 1]) * n + base[:, 0]
        grid = torch.zeros(n ** 3, 7, device=q.device, dtype=torch.float64)
        A = s["m"][:, None, None] * s["C"]
        S = -(4 * s["V"] / h ** 2)[:, None, None] * self.tau
        mv = s["m"][:, None] * s["v"]
        for i, j, k in off:
            wt = (w[:, i, 0] * w[:, j, 1] * w[:, k, 2])[:, None]
            dx = ((torch.tensor([i, j, k], device=q.device) - t) * h)[:, :, None]
            val = torch.cat([s["m"][:, None], mv + (A @ dx)[:, :, 0], (S @ dx)[:, :, 0]], 1)
            grid.index_add_(0, flat + (k * n + j) * n + i, wt * val)
        m = grid[:, :1]
        g = torch.tensor(self.d.gravity, device=q.device, dtype=torch.float64)
        u = torch.where(m > self.d.mass_eps, (grid[:, 1:4] + dt * (grid[:, 4:7] + m * g)) / torch.clamp(m, min=1e-300), 0 * m)
        u = u.reshape(n, n, n, 3)
        pos = self.o + torch.arange(n, device=q.device, dtype=torch.float64) * h
        low, high = pos < h * (1 - 1e-9), pos > (1 - h) * (1 + 1e-12)
        for a in range(3):
            shape = [1, 1, 1]
            shape[2 - a] = n
            c = u[..., a]
            u[..., a] = torch.where((low.reshape(shape) & (c < 0)) | (high.reshape(shape) & (c > 0)), 0 * c, c)
        u[:, low] = 0
        u = u.reshape(-1, 3)
        v, C = torch.zeros_like(s["v"]), torch.zeros_like(s["C"])
        for i, j, k in off:
            wt = (w[:, i, 0] * w[:, j, 1] * w[:, k, 2])[:, None]
            ui = wt * u[flat + (k * n + j) * n + i]
            v += ui
            C += ui[:, :, None] * (torch.tensor([i, j, k], device=q.device) - t)[:, None, :] * (4 / h)
        s["v"], s["C"] = v, C
        s["F"] = s["F"] + dt * C @ s["F"]
        s["x"] = torch.clamp(s["x"] + dt * v, 1e-6 * h, 1 - 1e-6 * h)
        self.tau = _law(self.mat, s, True, dt)

    def step(self, dt_requested, after=None):
        left, count = dt_requested, 0
        while left > 1e-6 * dt_requested and count < 48:
            dt = min(left, self.stable())
            if left - dt <= 1e-6 * dt_requested:
                dt = left
            self.substep(dt)
            if after:
                after(dt)
            left -= dt
            count += 1

    def out(self, fields):
        s, o = self.s, {}
        for f in fields:
            if f in "xv":
                for k, name in enumerate(("x", "y", "z") if f == "x" else ("vx", "vy", "vz")):
                    o[name] = s[f][:, k]
            elif f in "FC":
                o[f] = s[f].reshape(-1, 9)
            else:
                o[{"ep": "plastic", "T": "temperature"}[f]] = s[f]
        return o


def _pairs(x, radius):
    """All ordered pairs closer than radius, as index tensors, in pieces of i."""
    n = x.shape[0]
    order = torch.argsort(x[:, 2])
    xs = x[order]
    step = 2048
    for a in range(0, n, step):
        p = xs[a:a + step]
        lo = int(torch.searchsorted(xs[:, 2].contiguous(), p[0, 2] - radius))
        hi = int(torch.searchsorted(xs[:, 2].contiguous(), p[-1, 2] + radius))
        d = p[:, None, :] - xs[None, lo:hi, :]
        r = d.norm(dim=2)
        r[torch.arange(p.shape[0]), torch.arange(a, a + p.shape[0]) - lo] = math.inf
        i, j = torch.nonzero(r < radius, as_tuple=True)
        yield order[i + a], order[j + lo], d[i, j], r[i, j]


def _regularize(e, case, dt):
    s, k = e.s, _reg(case)
    t = k["spacing"] * torch.clamp(s["V"] * torch.linalg.det(s["F"]) / k["volume_unit"], 1 / 64, 8) ** (1 / 3)
    inv = 1 / s["m"]
    shift = torch.zeros_like(s["x"])
    gain = 1 - math.exp(-k["rate"] * dt)
    for i, j, d, r in _pairs(s["x"], float(t.max())):
        target = .5 * (t[i] + t[j])
        q = torch.where(r < target, (target - r) * gain / (r * (inv[i] + inv[j])), 0 * r)
        shift.index_add_(0, i, d * (q * inv[i])[:, None])
    over = max(1.0, float(shift.norm(dim=1).max()) / (k["max_speed"] * dt))
    s["x"] = torch.clamp(s["x"] + shift / over, 1e-6 * e.h, 1 - 1e-6 * e.h)


def _exact_heat(case, seed):
    i, mats, k, dt = _inputs(case, seed), _materials(case), _heat(case), _dt(case)
    pick = lambda f: torch.tensor([f(m) for m in mats], dtype=torch.float64, device=i["x"].device)[i["mat"]]  # noqa: E731
    cond, cp = pick(lambda m: m.conductivity), pick(lambda m: m.specific_heat)
    T, mcp = i["T"], _mass(i, mats) * cp
    gsum, heat = torch.zeros_like(T), torch.zeros_like(T)

    def g(a, b, r):
        return (1 - r / k["radius"]) * k["geometry"] * k["heat_rate"] * 2 * cond[a] * cond[b] / (cond[a] + cond[b])

    for a, b, _, r in _pairs(i["x"], k["radius"]):
        gsum.index_add_(0, a, g(a, b, r))
    budget = torch.where(gsum > 0, torch.clamp(.45 * mcp / (dt * torch.clamp(gsum, min=1e-300)), max=1), 1 + 0 * gsum)
    for a, b, _, r in _pairs(i["x"], k["radius"]):
        heat.index_add_(0, a, (T[b] - T[a]) * g(a, b, r) * dt * torch.minimum(budget[a], budget[b]))
    T = T + heat / mcp
    return {"temperature": T, "enthalpy": cp * T}


def _exact_plane(case, seed):
    """SolidMPM.frame of 1 / 60 s: substeps of min(left, stable step), gravity toward the centre, no wall within reach."""
    s = _plane_inputs(case, seed)
    n = s.count
    f = lambda a: torch.tensor(a[:n].astype(np.float64))  # noqa: E731
    x, v, m = torch.stack([f(s.x), f(s.y)], 1), torch.stack([f(s.vx), f(s.vy)], 1), f(s.mass)
    V, N, h, o = 12.96 * f(s.volume), 149, 8.0, -592.0
    F, C = torch.eye(2, dtype=torch.float64).expand(n, 2, 2).clone(), torch.zeros(n, 2, 2, dtype=torch.float64)
    mu = (.4 * m / V * 16000)[:, None, None]
    left, steps = 1 / 60, 0
    while left > 1e-9 and steps < 96:
        st = torch.clamp(F.reshape(n, 4).norm(dim=1), min=1)
        wave = max(1.0, float((v.norm(dim=1) + math.sqrt(19200) * st * st).max()))
        dt = min(left, 1 / 240, .18 * h / wave, .1 / max(1.0, float(C.abs().sum((1, 2)).max())))
        if case["gravity"] == "center":
            v = torch.clamp(v - x / torch.sqrt((x * x).sum(1, keepdim=True) + 400) * 27 * dt, -180, 180)
        q = (x - o) / h
        base = torch.clamp(torch.floor(q - .5).long(), 0, N - 3)
        t = q - base
        w = torch.stack([.5 * (1.5 - t) ** 2, .75 - (t - 1) ** 2, .5 * (t - .5) ** 2], 1)
        J = torch.linalg.det(F)[:, None, None]
        a, b = F[:, 0, 0] + F[:, 1, 1], F[:, 1, 0] - F[:, 0, 1]
        l = torch.sqrt(a * a + b * b)
        R = torch.stack([a / l, -b / l, b / l, a / l], 1).reshape(n, 2, 2)
        tau = 2 * mu * (F - R) @ F.transpose(1, 2) + mu * (J - 1) * J * torch.eye(2, dtype=torch.float64)
        A = m[:, None, None] * C - dt * (4 * V / h ** 2)[:, None, None] * tau
        grid = torch.zeros(N * N, 3, dtype=torch.float64)
        flat = base[:, 1] * N + base[:, 0]
        for j in range(3):
            for i in range(3):
                wt = (w[:, i, 0] * w[:, j, 1])[:, None]
                dx = ((torch.tensor([i, j]) - t) * h)[:, :, None]
                grid.index_add_(0, flat + j * N + i, wt * torch.cat([m[:, None], m[:, None] * v + (A @ dx)[:, :, 0]], 1))
        u = torch.where(grid[:, :1] > 1e-12, grid[:, 1:] / torch.clamp(grid[:, :1], min=1e-300), grid[:, 1:])
        v, C = torch.zeros_like(v), torch.zeros_like(C)
        for j in range(3):
            for i in range(3):
                ui = (w[:, i, 0] * w[:, j, 1])[:, None] * u[flat + j * N + i]
                v = v + ui
                C = C + ui[:, :, None] * (torch.tensor([i, j]) - t)[:, None, :] * (4 / h)
        F = F + dt * C @ F
        x = x + dt * v
        left -= dt
        steps += 1
    return [x[:, 0], x[:, 1], v[:, 0], v[:, 1]]


def exact(case, seed):
    kind = case["kind"]
    if kind == "plane":
        return _exact_plane(case, seed)
    if kind in ("batch", "soil"):
        return None
    n = _particles(case)
    if kind == "heat":
        return _exact_heat(case, seed)
    if kind == "run" and case["conduct"] or n * _substeps(case) > 3e7:
        return None
    e = _Exact(case, seed)
    for _ in range(case.get("steps", 1)):
        e.step(_dt(case), (lambda dt: _regularize(e, case, dt)) if kind == "regular" else None)
    if kind == "frame":
        return [e.s["x"][:, 0], e.s["x"][:, 1], e.s["x"][:, 2], e.s["v"][:, 0], e.s["v"][:, 1], e.s["v"][:, 2]]
    return e.out(_fields(case))
