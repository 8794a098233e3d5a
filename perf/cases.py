"""Measured workloads of the time step: what they are, their inputs, one pass, and their results in 64 bits.

A case is a dict of plain values:

  kind       "solve": a handle takes `steps` time steps and its state is read back
             "frame": a few steps, a display field and the read-outs of an interactive view
             "batch": `members` solves stepped together (`sizes`: one grid, or the four batched grid sizes)
  config     "plain" (cold-gas cone, inviscid), "viscous" (methalox bell with plume, viscous and reacting),
             "spray" (coaxial injector chamber with a parcel ring), or one of the engine presets
  nx, nr     grid;  steps  time steps of a pass;  precision  "fast" or "exact"

The flow a pass starts from is made from the seed: a quasi-one-dimensional nozzle solution with a boundary-layer
profile, an under- or over-expanded jet with a growing shear layer, and smooth disturbances; the chamber pressure
(for batches the ambient altitude too) follows the seed as well. Passes on one state continue the solve.
"""
import ctypes
import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = "rocket_nozzle_cfd_solver_b200"


def package():
    """The framework's package (its directory's name has dashes)."""
    if PKG not in sys.modules:
        d = os.path.join(ROOT, "rocket-nozzle-cfd-solver_b200")
        spec = importlib.util.spec_from_file_location(PKG, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        sys.modules[PKG] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[PKG])
    return sys.modules[PKG]


rn = package()
from rocket_nozzle_cfd_solver_b200 import configs, physics, simsetup, solver  # noqa: E402

SIZES = ((128, 48), (256, 96), (512, 192), (1024, 384))
PRESETS = ("demo", "overexp", "diamonds", "ideal", "underexp", "hybrid", "upper", "flight")
RING = 65536
LARGEST = 4096 * 1536 * 40


def solve(name, config, nx, nr, steps, precision="fast", parcels=0):
    return {"name": name, "kind": "solve", "config": config, "nx": nx, "nr": nr, "steps": steps,
            "precision": precision, "parcels": parcels}


def listed():
    return [
        # one step of the smallest grid, read back at once: a debugger's or an optimiser's inner call
        solve("single_step_128x48", "viscous", 128, 48, 1),
        # a lone solve of the smallest grid class of a study, 60 steps between two checks of its stop time
        solve("viscous_128x48", "viscous", 128, 48, 60),
        # the cold-gas cone of the parity workload
        solve("plain_256x96", "plain", 256, 96, 100),
        # the viscous plume of the headline benchmark
        solve("viscous_512x192", "viscous", 512, 192, 100),
        # the same in the precision that reproduces the oracle bit for bit
        solve("exact_512x192", "viscous", 512, 192, 50, precision="exact"),
        # the injector chamber with a full ring of 65,536 parcels
        solve("spray_512x192", "spray", 512, 192, 50, parcels=RING),
        # the app's medium grid (odd height) with an engine preset
        solve("preset_1024x287", "overexp", 1024, 287, 60),
        # a viscous grid beyond the L2 cache
        solve("viscous_2048x768", "viscous", 2048, 768, 60),
        # the largest grid of the benchmark, inviscid, resident in HBM
        solve("plain_4096x1536", "plain", 4096, 1536, 40),
        # one frame of the interactive view: steps, display field, wall row, exit column, chamber probe
        {"name": "frame_512x192", "kind": "frame", "config": "viscous", "nx": 512, "nr": 192, "steps": 8,
         "precision": "fast", "parcels": 0},
        # a study of 64 small nozzles stepped together
        {"name": "batch_64x128x48", "kind": "batch", "config": "viscous", "nx": 128, "nr": 48, "steps": 120,
         "members": 64, "precision": "fast"},
        # a study of nozzles over the four grid sizes
        {"name": "batch_24_mixed", "kind": "batch", "config": "viscous", "nx": 0, "nr": 0, "steps": 24,
         "members": 24, "precision": "fast"},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.2:
        c = {"kind": "batch", "config": "viscous", "nx": 0, "nr": 0, "steps": log_int(rng, 6, 120),
             "members": log_int(rng, 4, 64), "precision": "fast"}
        size = rng.choice((None,) + SIZES[:3])
        if size:
            c["nx"], c["nr"] = size
        while cells_of(c) * c["steps"] > LARGEST // 3:
            c["steps"] = max(1, c["steps"] // 2)
            c["members"] = max(4, c["members"] // 2)
        return c
    config = rng.choice(("plain", "viscous", "viscous", "spray") + PRESETS[:4] + PRESETS[4:])
    nx = log_int(rng, 256 if config == "spray" else 96, 1024 if config == "spray" else 2048)
    nr = max(24, int(round(nx * rng.uniform(0.25, 0.45))))
    frame = config != "spray" and rng.random() < 0.2
    c = {"kind": "frame" if frame else "solve", "config": config, "nx": nx, "nr": nr,
         "steps": log_int(rng, 1, 12) if frame else log_int(rng, 1, 120),
         "precision": "exact" if not frame and rng.random() < 0.15 else "fast",
         "parcels": log_int(rng, 2048, RING) if config == "spray" else 0}
    while cells_of(c) * c["steps"] > LARGEST // 3:
        c["steps"] = max(1, c["steps"] // 2)
    return c


def member_sizes(case):
    if case["kind"] != "batch":
        return [(case["nx"], case["nr"])]
    return [(case["nx"], case["nr"]) if case["nx"] else SIZES[m % 4] for m in range(case["members"])]


def cells_of(case):
    return sum(a * b for a, b in member_sizes(case))


# ---------------------------------------------------------------------------
# inputs
@functools.lru_cache(maxsize=48)
def setup_of(config, nx, nr, eps):
    """Grid and geometry (they do not depend on the seed); flow already started (no inlet ramp)."""
    if config == "plain":
        cfg = configs.plain_small(nx, nr)[0]
    elif config == "viscous":
        cfg = configs.viscous_plume(nx, nr)[0]
    elif config == "spray":
        cfg = configs.injector_spray(nx, nr)[0]
    else:
        cfg = configs.preset(config, nx, nr / nx)
    if eps:
        cfg["De"] = cfg["Dt"] * math.sqrt(eps)
    cfg["startMode"] = "burst"
    return rn.build_sim_setup(cfg)


def members_of(case, seed):
    """Per member: (setup, P, injector table or None, A, B) with A, B float32 [Nr, Nx, 4]."""
    rng = np.random.default_rng([int(seed) & 0x7fffffff, 77])
    out = []
    for m, (nx, nr) in enumerate(member_sizes(case)):
        batch = case["kind"] == "batch"
        s = setup_of(case["config"], nx, nr, (4.0, 9.0, 18.0, 40.0)[(m // 4 if case["nx"] == 0 else m) % 4] if batch else 0)
        cfg = dict(s.cfg, Pc=s.cfg["Pc"] * float(rng.uniform(0.9, 1.1)))
        if batch:
            cfg["alt"] = float(rng.uniform(0.0, 20e3))
        P = rn.compute_params(cfg, s.contour, s.dx, cfg["Pc"], physics.atmosphere(cfg["alt"])["p"])
        inj = simsetup.build_injector_table(cfg, s.contour, s.dx, P) if P["inj"] else None
        A, B = flow(s, P, rng)
        out.append((s, P, inj, A, B))
    return out


def smooth(rng, X, Y):
    """A smooth field of order 1 on the unit square coordinates X [Nx], Y [Nr]."""
    f = np.zeros((Y.size, X.size))
    for _ in range(5):
        kx, ky = rng.uniform(1.0, 14.0), rng.uniform(1.0, 8.0)
        f += 0.45 * (np.sin(2 * np.pi * ky * Y + rng.uniform(0, 6.3))[:, None] *
                     np.sin(2 * np.pi * kx * X + rng.uniform(0, 6.3))[None, :])
    return f


def flow(s, P, rng):
    Nx, Nr, dx, c = s.Nx, s.Nr, s.dx, s.contour
    g = P["gamma"]
    Ge, Ga = 1 / (g - 1), P["ambB"][2]
    rhoa, uinf, _, pa = P["amb"]
    Ta = pa / rhoa
    x = (np.arange(Nx) + 0.5) * dx
    r = (np.arange(Nr) + 0.5) * dx
    Rin = np.array([c.radiusAt(min(v, c.xe)) for v in x])
    # quasi-one-dimensional nozzle flow
    Ms = np.geomspace(0.005, 60.0, 4000)
    eps = (2 / (g + 1) * (1 + 0.5 * (g - 1) * Ms * Ms)) ** ((g + 1) / (2 * (g - 1))) / Ms
    sub = Ms <= 1
    ratio = np.maximum((Rin / c.Rt) ** 2, 1.0)
    M = np.where(x < c.xt, np.interp(ratio, eps[sub][::-1], Ms[sub][::-1]), np.interp(ratio, eps[~sub], Ms[~sub]))
    f = 1 + 0.5 * (g - 1) * M * M
    T1, p1 = P["res"][1] / f, P["res"][0] * f ** (-g / (g - 1))
    R = P["res"][2]
    u1 = M * np.sqrt(g * R * T1)
    slope = np.gradient(Rin, dx)
    # the jet: pressure swings about ambient along the axis and decays
    e = max(int(np.searchsorted(x, c.xe)) - 1, 0)
    sj = np.maximum(x - c.xe, 0.0) / c.Re
    out = x > c.xe
    swing = np.cos(2 * np.pi * sj / 3.0) * np.exp(-sj / 4.0)
    pj = np.where(out, pa * (p1[e] / pa) ** (0.7 * swing), p1)
    Tj = np.where(out, T1[e] * (pj / p1[e]) ** ((g - 1) / g), T1)
    uj = np.where(out, u1[e] * (1 - 0.05 * np.exp(-sj)), u1)
    Rj = np.where(out, c.Re * (1 + 0.1 * sj), Rin)
    w = np.where(out, 1.5 * dx + 0.08 * (x - c.xe), dx)
    b = np.where(out[None, :], 0.5 * (1 - np.tanh((r[:, None] - Rj[None, :]) / w[None, :])),
                 (r[:, None] < Rin[None, :]).astype(float))
    eta = np.minimum(r[:, None] / Rj[None, :], 1.0)
    shape = np.where(out[None, :], 1.0, 1 - 0.7 * eta ** 8)
    u = b * uj[None, :] * shape + (1 - b) * uinf
    v = b * uj[None, :] * shape * np.where(out, 0.05, slope)[None, :] * eta
    p = pa ** (1 - b) * pj[None, :] ** b
    T = b * Tj[None, :] + (1 - b) * Ta
    X, Y = x / x[-1], r / r[-1]
    u = u * (1 + 0.03 * smooth(rng, X, Y))
    v = v + 0.01 * np.abs(u) * smooth(rng, X, Y)
    p = p * (1 + 0.02 * smooth(rng, X, Y))
    T = T * (1 + 0.02 * smooth(rng, X, Y))
    Z = b
    F = Z * P["injData"]["Fres"] if P["inj"] else Z * (0.5 + 0.5 * b)
    Rm = (1 - Z) * P["RaN"] + F * P["Rs"][0] + np.maximum(Z - F, 0) * P["Rs"][2]
    G = b * Ge + (1 - b) * Ga
    rho = p / (Rm * T)
    A = np.stack((rho, rho * u, rho * v, p * G + 0.5 * rho * (u * u + v * v)), -1).astype(np.float32)
    B = np.stack((rho * Z, rho * F, G, np.zeros_like(G)), -1).astype(np.float32)
    if not P["inj"]:
        B[:, 0, 3] = P["uInlet0"]
    # merged cells hold their host's state; solid cells are ambient
    gm = np.asarray(s.geo["geoM"]).reshape(Nr, Nx, 4)
    solid = np.asarray(s.mask).reshape(Nr, Nx) != 0
    J, I = np.nonzero(((gm[..., 0] != 0) | (gm[..., 1] != 0)) & ~solid)
    Hj, Hi = J + gm[J, I, 1].astype(int), I + gm[J, I, 0].astype(int)
    A[J, I], B[J, I] = A[Hj, Hi], B[Hj, Hi]
    A[solid] = np.asarray(P["ambCons"], np.float32)
    B[solid] = np.asarray(P["ambB"], np.float32)
    return A, B


def parcels_of(case, s, P, inj, seed):
    """A ring holding case["parcels"] droplets spread over the chamber."""
    rng = np.random.default_rng([int(seed) & 0x7fffffff, 78])
    n = case["parcels"]
    tab = np.asarray(inj["tab"], np.float64).reshape(3, 256, 4)
    PA, PB = np.zeros((RING, 4), np.float32), np.zeros((RING, 4), np.float32)
    PA[:, :2] = -1
    row = rng.integers(0, 256, n)
    kind = tab[1, row, 0]
    PA[:n, 0] = rng.uniform(0.5, 0.8 * s.contour.xt / s.dx, n)
    PA[:n, 1] = np.sqrt(rng.uniform(0, 1, n)) * 0.9 * s.contour.Rc / s.dx
    PA[:n, 2] = rng.uniform(0.1, 0.5, n)
    PA[:n, 3] = rng.normal(0, 0.02, n)
    PB[:n, 0] = 50e-6 * np.exp(0.4 * rng.standard_normal(n))
    PB[:n, 1] = P["spray"]["mhat"] * 0.7 * P["cfl"] / P["wFloor"] / 4 * rng.uniform(0.3, 1.0, n)
    PB[:n, 2] = kind
    return PA, PB, n % RING


def prepare(case, seed):
    lib = solver.lib()
    state = {"case": case, "lib": lib, "members": [], "batch": None}
    if case["kind"] == "batch":
        state["batch"] = rn.SolverBatch()
    members = members_of(case, seed)
    if case["kind"] != "frame":   # the states come back into arrays of the caller's, members in turn
        state["A"], state["B"] = (torch.zeros(cells_of(case), 4, pin_memory=True) for _ in range(2))
        state["info"] = torch.zeros(len(members), 4, pin_memory=True)
    at = 0
    for k, (s, P, inj, A, B) in enumerate(members):
        h = rn.GPUSolver(s.Nx, s.Nr)
        if case["precision"] != "fast":
            h.setPrecision(case["precision"])
        h.setGeometry(s.geo)
        h.setState(A, B)
        if inj is not None:
            rn.GPUSpray(h).resize()
            h.spray.setInjector(inj)
            h.spray.setParcels(*parcels_of(case, s, P, inj, seed))
            state["PA"], state["PB"] = (torch.zeros(RING, 4, pin_memory=True) for _ in range(2))
        p = rn.params_from_P(P)
        m = {"solver": h, "P": p, "setup": s}
        if case["kind"] == "frame":
            m["spec"] = solver.derived_spec(dict(s, P=P), "mach", (0.0, 6.0))
            h.derived(m["spec"], p, read=False)
            m["field"] = torch.as_tensor(DeviceField(h, s.Nr, s.Nx), device="cuda")
        else:
            n = s.Nx * s.Nr
            m["to"] = (state["A"][at:].data_ptr(), state["B"][at:].data_ptr(),
                       ctypes.cast(state["info"][k].data_ptr(), ctypes.POINTER(ctypes.c_float)))
            at += n
        if state["batch"] is not None:
            state["batch"].add(h, p)
        state["members"].append(m)
    return state


class DeviceField:
    """The handle's display-field buffer as a CUDA array of Nr x Nx x 4 floats; keeps the handle alive."""

    def __init__(self, owner, nr, nx):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (nr, nx, 4), "typestr": "<f4", "version": 2,
                                         "data": (owner.derivedBuffer(), False)}


# ---------------------------------------------------------------------------
# one pass
def read_back(state):
    """The whole states (and the parcel ring) into the caller's pinned arrays."""
    lib, inj = state["lib"], False
    for m in state["members"]:
        h, (A, B, info) = m["solver"].h, m["to"]
        rc = lib.rn_get_state(h, A, B) or lib.rn_read_step_info(h, info)
        if m["P"].inj:
            inj = True
            for k, tex in (("PA", solver.RN_TEX_PARCEL_A), ("PB", solver.RN_TEX_PARCEL_B)):
                rc = rc or lib.rn_read_rect(h, tex, 0, 0, 256, 256, state[k].data_ptr())
        if rc:
            raise RuntimeError(lib.rn_last_error().decode())
    return outputs_of(state["A"], state["B"], state["info"], state.get("PA"), state.get("PB"), inj)


def outputs_of(A, B, info, PA, PB, inj):
    """Field by field over the cells, members in turn."""
    o = {"rho": A[:, 0], "rhou": A[:, 1], "rhov": A[:, 2], "E": A[:, 3], "rhoZ": B[:, 0], "rhoF": B[:, 1],
         "G": B[:, 2], "dt": info[:, 0], "t": info[:, 2]}
    # oxidiser density with an injector, else the mean inlet speed kept in the first column
    o["rhoO" if inj else "ubar"] = B[:, 3]
    if PA is not None:
        o["parcels"], o["droplets"], o["mass"] = PA, PB[:, 0], PB[:, 1]
    return o


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return read_back(state)
    m = state["members"][0]
    m["solver"].step(case["steps"], m["P"])
    return read_back(state) if case["kind"] == "solve" else frame(m)


def frame(m):
    g, s = m["solver"], m["setup"]
    g.derived(m["spec"], m["P"], read=False)
    row = g.drawWallRow()
    g.requestAsync([{"name": "info", "tex": g.stepInfoTex, "x": 0, "y": 0, "w": 1, "h": 1},
                    {"name": "A", "tex": g.state["A"], "x": s.iExit, "y": 0, "w": 1, "h": s.Nr},
                    {"name": "B", "tex": g.state["B"], "x": s.iExit, "y": 0, "w": 1, "h": s.Nr},
                    {"name": "probe", "tex": g.state["A"], "x": s.iChamber, "y": 0, "w": 1, "h": 1},
                    {"name": "wall", "tex": row, "x": 0, "y": 0, "w": s.Nx, "h": 1}], 1)
    got = None
    while got is None:
        got = g.pollAsync()
    d = got["data"]
    return {"field": m["field"], "dt": d["info"][0:1], "t": d["info"][2:3], "A": d["A"], "B": d["B"],
            "probe": d["probe"], "wall": d["wall"]}


# ---------------------------------------------------------------------------
# what a pass needs and how close two correct implementations come
def work(case):
    """Per cell and step: the state read and written once (64 bytes) and the geometry read (49); about 1,300
    operations (two stages of two faces a cell, the group update), 1,600 with the viscous and reacting terms.
    Per live parcel and step 64 bytes and 150 operations."""
    n = cells_of(case) * case["steps"]
    parcels = case.get("parcels", 0) * case["steps"]
    return {"bytes": 113.0 * n + 64.0 * parcels,
            "flops": (1300.0 if case["config"] == "plain" else 1600.0) * n + 150.0 * parcels}


def tolerance(case):
    """Rounding of 32-bit arithmetic carried through the steps of a pass: shocks, limiters and the shear layer
    amplify it, most in the small transverse momentum (8e-6 off 64 bits after 60 steps of 1024 x 287). With
    parcels the oxidiser vapour, a small sum of source terms, is 2e-4 off."""
    return {"rel": 1e-3 if case["config"] == "spray" else 5e-5}


# ---------------------------------------------------------------------------
# the same in 64 bits
RHO_MIN = P_MIN = 1e-7


def clip(x, lo, hi):
    return torch.minimum(torch.maximum(x, lo if torch.is_tensor(lo) else torch.full_like(x, lo)),
                         hi if torch.is_tensor(hi) else torch.full_like(x, hi))


def smoothstep(e0, e1, x):
    t = ((x - e0) / (e1 - e0)).clamp(0.0, 1.0)
    return t * t * (3 - 2 * t)


def mix(a, b, f):
    return a * (1 - f) + b * f


class Exact:
    """The time step of the members of one grid size, [member, row, column] planes of doubles."""

    def __init__(self, members):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        s0, P0 = members[0][0], members[0][1]
        self.Nx, self.Nr, self.n, self.dev = s0.Nx, s0.Nr, len(members), dev
        n, Nx, Nr = self.n, self.Nx, self.Nr
        self.inj, self.visc, self.chem, self.order2 = (bool(P0[k]) for k in ("inj", "visc", "chem", "order2"))
        stack = lambda k, *sh: torch.stack([f64(m[0].geo[k]).reshape(sh) for m in members])  # noqa: E731
        geoA, geoG, gm = stack("geoA", Nr + 1, Nx + 1, 4), stack("geoG", Nr, Nx, 4), stack("geoM", Nr, Nx, 4)
        self.solid = torch.stack([f64(m[0].mask).reshape(Nr, Nx) != 0 for m in members])
        self.ax, self.ar = geoA[:, :Nr, :, 2].contiguous(), geoA[:, :, :Nx, 3].clone()
        self.ar[:, 0] = 0.0
        self.gV, self.gAm, self.gWx, self.gWr = (geoG[..., k].contiguous() for k in range(4))
        hx, hy = gm[..., 0].round().long(), gm[..., 1].round().long()
        hx, hy = hx.masked_fill(self.solid, 0), hy.masked_fill(self.solid, 0)
        J, I = torch.meshgrid(torch.arange(Nr, device=dev), torch.arange(Nx, device=dev), indexing="ij")
        self.J, self.I = J.double(), I.double()
        base = (torch.arange(n, device=dev) * (Nr * Nx)).view(n, 1, 1)
        self.host = base + (J + hy) * Nx + (I + hx)
        self.base = base
        self.bits = gm[..., 2].round().long().masked_fill(self.solid, 0)
        self.band = ((self.bits & 16) != 0).double()
        self.bits = [((self.bits & k) != 0).double() for k in (1, 2, 4, 8)]
        self.l = gm[..., 3].contiguous()
        p32 = lambda f: f64([np.float32(f(m[1])) for m in members]).view(n, 1, 1)  # noqa: E731
        self.p = {k: p32(lambda P, k=k: P[k]) for k in ("Tw", "cfl", "dtMax", "wFloor", "vMax", "hllBlend", "pStart",
                                                       "RcCells")}
        for k in ("amb", "ambCons", "ambB", "gamR", "inlet", "res", "gas", "Rs", "chemK", "cap", "chamberNu"):
            self.p[k] = [p32(lambda P, k=k, q=q: P[k][q]) for q in range(len(P0[k]))]
        self.p["barMax"] = p32(lambda P: 1.6 * P["uInlet0"])
        self.A = torch.stack([f64(m[3]) for m in members]).permute(3, 0, 1, 2).contiguous()
        self.B = torch.stack([f64(m[4]) for m in members]).permute(3, 0, 1, 2).contiguous()
        z = torch.zeros(n, 1, 1, dtype=torch.float64, device=dev)
        self.dt, self.t, self.first = z, z.clone(), True

    def at_host(self, x):
        return x.reshape(-1)[self.host]

    @staticmethod
    def prims(A, B):
        rho = A[0].clamp(min=RHO_MIN)
        u, v, G = A[1] / rho, A[2] / rho, B[2].clamp(min=0.5)
        p = ((A[3] - 0.5 * rho * (u * u + v * v)) / G).clamp(min=P_MIN)
        return [rho, u, v, p, (B[0] / rho).clamp(0, 1), (B[1] / rho).clamp(0, 1), G, (B[3] / rho).clamp(0, 1)]

    @staticmethod
    def sound(q):
        return torch.sqrt((1 + 1 / q[6]) * q[3] / q[0])

    def pad(self, A, B):
        """Primitives with two ghost cells all round, and the wall flags."""
        n, Nx, Nr, p = self.n, self.Nx, self.Nr, self.p
        q = self.prims(A, B)
        Q = torch.zeros(8, n, Nr + 4, Nx + 4, dtype=torch.float64, device=self.dev)
        S = torch.zeros(n, Nr + 4, Nx + 4, dtype=torch.bool, device=self.dev)
        amb = [*p["amb"], torch.zeros_like(self.dt), torch.zeros_like(self.dt), p["inlet"][3], torch.zeros_like(self.dt)]
        for k in range(8):
            Q[k, :, 2:Nr + 2, 2:Nx + 2] = q[k]
        S[:, 2:Nr + 2, 2:Nx + 2] = self.solid
        # right edge, then the top (with the corner): supersonic outflow copies, subsonic outflow takes ambient pressure
        e = [k[:, :, -1:] for k in q]
        out, sup, sol = e[1] > 0, e[1] >= self.sound(e), self.solid[:, :, -1:]
        for k in range(8):
            a = amb[k].clamp(min=0) if k == 1 else amb[k]
            v = torch.where(sup, e[k], torch.where(out, amb[k] if k == 3 else e[k], a))
            Q[k, :, 2:Nr + 2, Nx + 2:] = torch.where(sol, amb[k], v)
        e = [torch.cat([k[:, -1:, :], k[:, -1:, -1:], k[:, -1:, -1:]], 2) for k in q]
        sol = torch.cat([self.solid[:, -1:, :], self.solid[:, -1:, -1:], self.solid[:, -1:, -1:]], 2)
        out, sup = e[2] > 0, e[2] >= self.sound(e)
        for k in range(8):
            v = torch.where(sup, e[k], torch.where(out, amb[k] if k == 3 else e[k], amb[k]))
            Q[k, :, Nr + 2:, 2:] = torch.where(sol, amb[k], v)
        # left edge: inlet below the chamber radius, wall where the first column is solid, ambient above
        rows = torch.arange(Nr + 2, device=self.dev).double().view(1, -1, 1) + 0.5
        chamber = rows < p["RcCells"]
        wall = torch.cat([self.solid[:, :, :1], torch.zeros(n, 2, 1, dtype=torch.bool, device=self.dev)], 1)
        if self.inj:
            wall = wall | chamber
        T0, R, G = p["res"][1], p["res"][2], p["inlet"][2]
        gg = 1 + 1 / G
        c0 = torch.sqrt(gg * R * T0)
        u0 = (A[1][:, :, :1] / A[0][:, :, :1].clamp(min=RHO_MIN))
        ui = torch.minimum(u0.clamp(min=0), 0.5 * c0)
        ut = B[3][:, :, :1].clamp(min=0) * smoothstep(1.0, 2.0, p["res"][0] / p["pStart"].clamp(min=1e-6))
        u = mix(ui, ut, p["inlet"][1])
        T = T0 - u * u * (gg - 1) / (2 * gg * R)
        pr = p["res"][0] * (T / T0) ** (gg * G)
        one = torch.ones_like(u)
        inlet = [pr / (R * T), u, 0 * one, pr, one, one, G * one, 0 * one]
        for k in range(8):
            v = torch.cat([inlet[k], amb[k].expand(n, 2, 1)], 1)
            Q[k, :, 2:, :2] = torch.where(chamber, v, amb[k])
        S[:, 2:, :2] = wall
        # the axis mirrors
        for a, b in ((1, 2), (0, 3)):
            Q[:, :, a], S[:, a] = Q[:, :, b], S[:, b]
            Q[2, :, a] = -Q[2, :, a]
        return Q, S

    def flux(self, w, S, sides, area, r_dir):
        """Flux of a set of faces: w the four cells along the normal (8 planes each), S their wall flags, sides
        the pressure and flag of the cells beside the inner two."""
        p = self.p
        w = [[x for x in c] for c in w]
        if r_dir:
            for c in w:
                c[1], c[2] = c[2], c[1]
        s0, s1, s2, s3 = S
        jm = torch.zeros_like(area)
        for pc, near in ((w[1][3], sides[0:2]), (w[2][3], sides[2:4])):
            for ps, ss in near:
                ps = torch.where(ss, pc, ps)
                jm = torch.maximum(jm, (ps - pc).abs() / torch.minimum(ps, pc))
        blend = smoothstep(0.15, 0.6, jm * p["hllBlend"]).masked_fill(s1 | s2, 0.0)

        def mirror(c, k):
            return -c[k] if k == 1 else c[k]

        lo = [torch.where(s0, mirror(w[1], k), w[0][k]) for k in range(8)]
        hi = [torch.where(s3, mirror(w[2], k), w[3][k]) for k in range(8)]

        def limit(a, b):
            ab, den = a * b, a + b
            return 2 * ab.clamp(min=0) / torch.where(den.abs() > 1e-30, den, torch.ones_like(den))

        L, R = [], []
        for k in range(8):
            d = w[2][k] - w[1][k]
            L.append(w[1][k] + 0.5 * limit(w[1][k] - lo[k], d))
            R.append(w[2][k] - 0.5 * limit(d, hi[k] - w[2][k]))
        second = (area > 0) & ~s1 & ~s2 & (L[0] > 0) & (L[3] > 0) & (R[0] > 0) & (R[3] > 0)
        if not self.order2:
            second = torch.zeros_like(second)
        for c, v in ((L, w[1]), (R, w[2])):
            for k in (4, 5, 7):
                c[k] = c[k].clamp(0, 1)
            c[6] = c[6].clamp(0.5, 100.0)
            for k in range(8):
                c[k] = torch.where(second, c[k], v[k])
        for k in range(8):
            L[k], R[k] = (torch.where(s1, mirror(w[2], k), L[k]), torch.where(s2 & ~s1, mirror(w[1], k), R[k]))
            R[k] = torch.where(s1, w[2][k], R[k])
        rL, uL, vL, pL, ZL, FL, GL, OL = L
        rR, uR, vR, pR, ZR, FR, GR, OR = R
        cL, cR = self.sound(L), self.sound(R)
        EL, ER = pL * GL + 0.5 * rL * (uL * uL + vL * vL), pR * GR + 0.5 * rR * (uR * uR + vR * vR)
        a, b = torch.sqrt(rL), torch.sqrt(rR)
        a, b = a / (a + b), b / (a + b)
        uT, vT, GT = a * uL + b * uR, a * vL + b * vR, a * GL + b * GR
        HT = a * (EL + pL) / rL + b * (ER + pR) / rR
        cT = torch.sqrt(((HT - 0.5 * (uT * uT + vT * vT)) / GT).clamp(min=1e-12))
        SL, SR = torch.minimum(uL - cL, uT - cT), torch.maximum(uR + cR, uT + cT)
        mL, mR = rL * uL, rR * uR
        one = torch.ones_like(rL)
        UL, UR = [rL, mL, rL * vL, EL, rL * ZL, rL * FL, rL * OL], [rR, mR, rR * vR, ER, rR * ZR, rR * FR, rR * OR]
        fL = [mL, mL * uL + pL, mL * vL, uL * (EL + pL), mL * ZL, mL * FL, mL * OL]
        fR = [mR, mR * uR + pR, mR * vR, uR * (ER + pR), mR * ZR, mR * FR, mR * OR]
        Ss = (pR - pL + mL * (SL - uL) - mR * (SR - uR)) / (rL * (SL - uL) - rR * (SR - uR))
        left = Ss >= 0
        pick = lambda x, y: torch.where(left, x, y)  # noqa: E731
        rK, uK, vK, pK, EK, SK = pick(rL, rR), pick(uL, uR), pick(vL, vR), pick(pL, pR), pick(EL, ER), pick(SL, SR)
        kk = rK * (SK - uK) / (SK - Ss)
        star = [kk, kk * Ss, kk * vK, kk * (EK / rK + (Ss - uK) * (Ss + pK / (rK * (SK - uK)))), kk * pick(ZL, ZR),
                kk * pick(FL, FR), kk * pick(OL, OR)]
        inv, SLR = 1 / (SR - SL), SL * SR
        out = []
        for k in range(7):
            c = pick(fL[k], fR[k]) + SK * (star[k] - pick(UL[k], UR[k]))
            h = (SR * fL[k] - SL * fR[k] + SLR * (UR[k] - UL[k])) * inv
            f = torch.where(blend > 0, mix(c, h, blend), c)
            out.append(torch.where(SL >= 0, fL[k], torch.where(SR <= 0, fR[k], f)))
        uf = uK + SK * ((SK - uK) / (SK - Ss) - 1)
        uf = torch.where(SL >= 0, uL, torch.where(SR <= 0, uR, uf))
        Gf = torch.where(SL >= 0, GL, torch.where(SR <= 0, GR, pick(GL, GR)))
        if r_dir:
            out[1], out[2] = out[2], out[1]
        out = out[:6] + [uf * Gf, uf, out[6]]
        open_ = (area != 0) & ~(s1 & s2)
        return [torch.where(open_, x * one, torch.zeros_like(x)) for x in out]

    def member_sum(self, fx, fr):
        """Area-weighted net flux of each cell plus that of its slaves, read at each cell's host."""
        ax, ar = self.ax.abs(), self.ar.abs()
        out = []
        for x, r in zip(fx, fr):
            gx, gr = ax * x, ar * r
            m = -(gx[:, :, 1:] - gx[:, :, :-1]) - (gr[:, 1:] - gr[:, :-1])
            s = m.clone()
            s[:, :, 1:] += self.bits[0][:, :, 1:] * m[:, :, :-1]
            s[:, :, :-1] += self.bits[1][:, :, :-1] * m[:, :, 1:]
            s[:, 1:] += self.bits[2][:, 1:] * m[:, :-1]
            s[:, :-1] += self.bits[3][:, :-1] * m[:, 1:]
            out.append(self.at_host(s))
        return out

    def net_flux(self, Q, S):
        Nx, Nr = self.Nx, self.Nr
        r, c = slice(2, Nr + 2), slice(2, Nx + 2)
        cols = [slice(k, Nx + 1 + k) for k in range(4)]
        side = lambda a, b: (Q[3][:, a, b], S[:, a, b])  # noqa: E731
        up, dn = slice(3, Nr + 3), slice(1, Nr + 1)
        fx = self.flux([Q[:, :, r, k] for k in cols], [S[:, r, k] for k in cols],
                       [side(up, cols[1]), side(dn, cols[1]), side(up, cols[2]), side(dn, cols[2])], self.ax, False)
        rows = [slice(k, Nr + 1 + k) for k in range(4)]
        ea, we = slice(3, Nx + 3), slice(1, Nx + 1)
        fr = self.flux([Q[:, :, k, c] for k in rows], [S[:, k, c] for k in rows],
                       [side(rows[1], ea), side(rows[1], we), side(rows[2], ea), side(rows[2], we)], self.ar, True)
        return self.member_sum(fx, fr)

    def fill_solid(self, A, B):
        for k in range(4):
            A[k] = torch.where(self.solid, self.p["ambCons"][k], A[k])
            B[k] = torch.where(self.solid, self.p["ambB"][k], B[k])
        return torch.stack(A), torch.stack(B)

    def stage(self, A, B, A0, B0, dt, t, second):
        p = self.p
        Q, S = self.pad(A, B)
        L = self.net_flux(Q, S)
        Ah, Bh = [self.at_host(x) for x in A], [self.at_host(x) for x in B]
        q = self.prims(Ah, Bh)
        Wx, Wr, wl = self.gWx, self.gWr, torch.sqrt(self.gWx ** 2 + self.gWr ** 2)
        near = wl > 1e-6
        wls = torch.where(near, wl, torch.ones_like(wl))
        un = (q[1] * Wx + q[2] * Wr) / wls
        g = 1 + 1 / q[6]
        c = torch.sqrt(g * q[3] / q[0])
        a = 0.25 * (g + 1) * un
        press = q[3] + q[0] * un * (a + torch.sqrt(a * a + c * c))
        suct = q[3] * (1 + 0.5 * (g - 1) * un / c).clamp(min=0) ** (2 * g / (g - 1))
        pw = torch.where(un > 0, press, suct).masked_fill(~near, 0.0)
        L[1], L[2] = L[1] - Wx * pw, L[2] - Wr * pw + q[3] * self.gAm
        f = dt / self.gV.clamp(min=1e-6)
        LA = L[0:4]
        LB = [L[4], L[5], L[6] - q[6] * L[7], L[8]]
        U, Y = [Ah[k] + f * LA[k] for k in range(4)], [Bh[k] + f * LB[k] for k in range(4)]
        if second:
            U = [0.5 * (self.at_host(A0[k]) + U[k]) for k in range(4)]
            Y = [0.5 * (self.at_host(B0[k]) + Y[k]) for k in range(4)]
        rho = U[0].clamp(min=RHO_MIN)
        vx, vy = U[1] / rho, U[2] / rho
        sp = torch.sqrt(vx * vx + vy * vy)
        s = torch.where(sp > p["vMax"], p["vMax"] / sp.clamp(min=1e-30), torch.ones_like(sp))
        vx, vy = vx * s, vy * s
        G = clip(Y[2], p["gamR"][0], p["gamR"][1])
        E = torch.maximum(U[3], P_MIN * G + 0.5 * rho * (vx * vx + vy * vy))
        Z = clip(Y[0], 0.0, rho)
        if self.inj:
            w = clip(Y[3], 0.0, rho)
        else:
            w = torch.zeros_like(rho)
            u0 = B[3][:, :, 0]
            if second:
                bar = torch.minimum(u0 + (dt * p["inlet"][0]).clamp(max=1.0)[:, :, 0] * (vx[:, :, 0] - u0), p["barMax"][:, :, 0])
                u0 = torch.where(t[:, :, 0] > 0, bar, u0)
            w[:, :, 0] = u0
        A2, B2 = self.fill_solid([rho, rho * vx, rho * vy, E], [Z, clip(Y[1], 0.0, Z), G, w])
        return A2, B2, Q, S

    def gas_constant(self, s):
        p = self.p
        return ((1 - s[4]) * p["gas"][0] + s[5] * p["Rs"][0] + s[7] * p["Rs"][1] +
                (s[4] - s[5] - s[7]).clamp(min=0) * p["Rs"][2])

    def sutherland(self, TK):
        return self.p["gas"][3] * 1.458e-6 * TK * torch.sqrt(TK) / (TK + 110.4)

    def viscosity(self, Q, S, dt):
        """Velocity gradients, effective viscosity, enthalpy and filtered strain of the cells."""
        p, Nx, Nr = self.p, self.Nx, self.Nr
        r, c = slice(2, Nr + 2), slice(2, Nx + 2)
        q = [Q[k][:, r, c] for k in range(8)]
        E, W = (slice(None), r, slice(3, Nx + 3)), (slice(None), r, slice(1, Nx + 1))
        N, D = (slice(None), slice(3, Nr + 3), c), (slice(None), slice(1, Nr + 1), c)
        ok = {k: (~S[i]).double() for k, i in (("E", E), ("W", W), ("N", N), ("D", D))}
        nx, nr = (ok["E"] + ok["W"]).clamp(min=1), (ok["N"] + ok["D"]).clamp(min=1)
        dx = lambda k: (ok["E"] * (Q[k][E] - q[k]) + ok["W"] * (q[k] - Q[k][W])) / nx  # noqa: E731
        dr = lambda k: (ok["N"] * (Q[k][N] - q[k]) + ok["D"] * (q[k] - Q[k][D])) / nr  # noqa: E731
        ux, vx, ur, vr = dx(1), dx(2), dr(1), dr(2)
        vor = q[2] / (self.J + 0.5)
        div = ux + vr + vor
        S2 = 2 * (ux * ux + vr * vr + vor * vor) + (ur + vx) ** 2 - 0.6666667 * div * div
        om = vx - ur
        strain = torch.sqrt(S2.clamp(min=0)) * (om * om / (om * om + div * div + 1e-8))
        mu = self.sutherland(q[3] / (q[0] * self.gas_constant(q)) * p["gas"][2])
        mut = q[0] * self.l * self.l * strain
        mut = torch.where(self.I < p["chamberNu"][1], torch.maximum(mut, q[0] * p["chamberNu"][0]), mut)
        eff = torch.minimum(mu + mut, 0.08 * q[0] / dt.clamp(min=1e-9))
        T = [ux, ur, vx, vr, eff, (q[6] + 1) * q[3] / q[0], strain, mu]
        return [x.masked_fill(self.solid, 0.0) for x in T]

    def viscous_flux(self, Q, S, T, r_dir):
        Nx, Nr = self.Nx, self.Nr
        a = (slice(None), slice(2, Nr + 2), slice(2, Nx + 2))
        q = [Q[k][a] for k in range(8)]
        s = S[a]
        if r_dir:
            one, two = (slice(None), slice(0, Nr - 1), slice(None)), (slice(None), slice(1, Nr), slice(None))
            r = torch.arange(1, Nr, device=self.dev).double().view(1, -1, 1)
            area = self.ar[:, 1:Nr]
        else:
            one, two = (slice(None), slice(None), slice(0, Nx - 1)), (slice(None), slice(None), slice(1, Nx))
            r = torch.arange(Nr, device=self.dev).double().view(1, -1, 1) + 0.5
            area = self.ax[:, :, 1:Nx]
        mid = lambda x: 0.5 * (x[one] + x[two])  # noqa: E731
        d = lambda x: x[two] - x[one]  # noqa: E731
        mu, uf, vf = mid(T[4]), mid(q[1]), mid(q[2])
        ux, vx, ur, vr = (mid(T[0]), mid(T[2]), d(q[1]), d(q[2])) if r_dir else (d(q[1]), d(q[2]), mid(T[1]), mid(T[3]))
        div = ux + vr + vf / r
        txr, k = mu * (ur + vx), mu * 1.25
        if r_dir:
            trr = mu * (2 * vr - 0.6666667 * div)
            f = [-k * d(q[7]), -txr, -trr, -(uf * txr + vf * trr) - k * d(T[5])]
        else:
            txx = mu * (2 * ux - 0.6666667 * div)
            f = [-k * d(q[7]), -txx, -txr, -(uf * txx + vf * txr) - k * d(T[5])]
        f += [-k * d(q[4]), -k * d(q[5]), -k * d(q[6])]
        shut = s[one] | s[two] | (area == 0)
        pad = (0, 0, 1, 1) if r_dir else (1, 1)
        return [torch.nn.functional.pad(x.masked_fill(shut, 0.0), pad) for x in f]

    def source(self, A, B, Q, S, dt):
        p, Nx, Nr = self.p, self.Nx, self.Nr
        T = self.viscosity(Q, S, dt)
        Ah, Bh = [self.at_host(x) for x in A], [self.at_host(x) for x in B]
        q = self.prims(Ah, Bh)
        rho, u, v, pr, Z, F, G, O = q
        V = self.gV.clamp(min=1e-6)
        Rm = self.gas_constant(q)
        Tg = pr / (rho * Rm)
        Th = [self.at_host(x) for x in T]
        L = [torch.zeros_like(rho)] * 7
        if self.visc:
            L = self.member_sum(self.viscous_flux(Q, S, T, False), self.viscous_flux(Q, S, T, True))
            vor = v / (V / self.gAm.clamp(min=1e-6))
            L[2] = L[2] - Th[4] * (2 * vor - 0.6666667 * (Th[0] + Th[3] + vor)) * self.gAm
            # wall shear and heat flux
            wl = torch.sqrt(self.gWx ** 2 + self.gWr ** 2)
            near = wl > 1e-6
            wl = torch.where(near, wl, torch.ones_like(wl))
            nx, nr = self.gWx / wl, self.gWr / wl
            dn = u * nx + v * nr
            ux, ur = u - dn * nx, v - dn * nr
            up = torch.sqrt(ux * ux + ur * ur)
            cp = Rm * (G + 1)
            Taw = Tg + 0.89 * up * up / (2 * cp)
            Ts = (Tg + 0.5 * (p["Tw"] - Tg) + 0.22 * (Taw - Tg)).clamp(min=1e-3)
            rs, mus = pr / (Rm * Ts), self.sutherland(Ts * p["gas"][2])
            dz = 2 * (0.5 * V / wl).clamp(0.25, 1.0)
            nz = mus / (rs * dz)
            turb = rs * (7.187 * nz ** 1.142857 + 0.13769 * nz ** 0.142857 * up) ** 1.75
            tw = torch.where(up <= 69.7 * nz, 2 * mus * up / dz, turb)
            tw = torch.minimum(tw, 0.3 * rho * up * V / (wl * dt).clamp(min=1e-9))
            pull = torch.where(near & (up > 1e-6), tw * wl / up.clamp(min=1e-30), torch.zeros_like(tw))
            L[1], L[2] = L[1] - pull * ux, L[2] - pull * ur
            qw = tw / up.clamp(min=1e-4) * cp * (Taw - p["Tw"]) * 1.24
            qm = 0.3 * pr * G * V / (wl * dt).clamp(min=1e-9)
            L[3] = L[3] - (torch.minimum(torch.maximum(qw, -qm), qm) * wl).masked_fill(~near, 0.0)
            # separation: pressure sampled downstream in the wall band
            sp = torch.sqrt(u * u + v * v)
            Mn = sp / torch.sqrt((1 + 1 / G) * pr / rho)
            hj, hi = (self.host - self.base) // Nx, (self.host - self.base) % Nx
            sx, sr = u / sp.clamp(min=1e-30), v / sp.clamp(min=1e-30)
            gas = torch.where(S, torch.zeros_like(Q[3]), Q[3])[:, 2:Nr + 2, 2:Nx + 2].reshape(-1)
            pd = torch.zeros_like(rho)
            for n in (4, 6):
                for m in (0, 1):
                    i = (hi + torch.round(n * sx).long()).clamp(0, Nx - 1)
                    j = (hj + torch.floor(n * sr).long() + m).clamp(0, Nr - 1)
                    pd = torch.maximum(pd, gas[self.base + j * Nx + i])
            crit = 1 + 0.5 * Mn
            fs = smoothstep(crit, 1.2 * crit, pd / pr) * V * rho * sp
            slow = (u > 0) & (pr < 1.3 * p["chemK"][3])
            fs = torch.where(Mn > 1, fs, torch.where(slow, 0.5 * V * rho * sp, torch.zeros_like(fs)))
            fs = fs * self.at_host(self.band)
            L[1], L[2] = L[1] - fs * u, L[2] - fs * v
        f = dt / V
        U = [Ah[0], Ah[1] + f * L[1], Ah[2] + f * L[2], Ah[3] + f * L[3]]
        Y = [Bh[0] + f * L[4], Bh[1] + f * L[5], Bh[2] + f * L[6] / rho, Bh[3]]
        if self.inj:
            Y[3] = Y[3] + f * L[0]
        if self.chem:
            s = p["chemK"][1]
            air = (1 - Z).clamp(min=0) if self.inj else None
            avail = torch.minimum(F, (O + 0.233 * air) / s if self.inj else (1 - Z - s * (Z - F)).clamp(min=0) / s)
            TK = Tg * p["gas"][2]
            kin = p["chemK"][2] * pr * torch.exp(-9000.0 / TK) * (1 - smoothstep(p["cap"][0], p["cap"][1], TK))
            mixing = torch.maximum(Th[6], 4 * Th[4] / rho) if self.inj else Th[6]
            burn = rho * avail * (torch.minimum(mixing, kin) * dt).clamp(max=0.5)
            burn = burn.masked_fill(avail <= 1e-5, 0.0)
            Y[1] = Y[1] - burn
            if self.inj:
                Y[3] = torch.where(avail > 1e-5, (Y[3] - burn * s).clamp(min=0), Y[3])
            U[3] = U[3] + burn * p["chemK"][0]
        rn_ = U[0].clamp(min=RHO_MIN)
        vx, vy = U[1] / rn_, U[2] / rn_
        G2 = clip(Y[2], p["gamR"][0], p["gamR"][1])
        Z2 = clip(Y[0], 0.0, rn_)
        E = torch.maximum(U[3], P_MIN * G2 + 0.5 * rn_ * (vx * vx + vy * vy))
        return self.fill_solid([rn_, rn_ * vx, rn_ * vy, E],
                               [Z2, clip(Y[1], 0.0, Z2), G2, clip(Y[3], 0.0, rn_) if self.inj else B[3].clone()])

    def step(self):
        p = self.p
        q = self.prims(self.A, self.B)
        w = (q[1].abs() + q[2].abs() + 2 * self.sound(q)).masked_fill(self.solid, 0.0).amax((1, 2), keepdim=True)
        dt = torch.minimum(p["cfl"] / torch.maximum(p["wFloor"], w), p["dtMax"])
        if not self.first:
            dt = torch.minimum(dt, 1.2 * self.dt)
        self.first, self.dt = False, dt
        self.t = self.t + dt
        A1, B1, _, _ = self.stage(self.A, self.B, None, None, dt, self.t - dt, False)
        A2, B2, Q, S = self.stage(A1, B1, self.A, self.B, dt, self.t, True)
        if self.visc or self.chem:
            A2, B2 = self.source(A2, B2, Q, S, dt)
        self.A, self.B = A2, B2
        return Q, S


class ExactSpray:
    """The parcel ring of one injector chamber, in 64 bits (fields as in the ring: PA = x, r, u, v; PB = d, m, type, xi)."""

    def __init__(self, ex, P, inj, PA, PB, head):
        f = lambda a: torch.as_tensor(np.asarray(a, np.float32).astype(np.float64), device=ex.dev)  # noqa: E731
        self.ex, self.PA, self.PB, self.head, self.seed = ex, f(PA), f(PB), head, 1
        self.tab = f(np.asarray(inj["tab"]).reshape(3, 256, 4))
        d, one = P["injData"], lambda v: float(np.float32(v))  # noqa: E731
        self.mhat, self.tScale = one(P["spray"]["mhat"]), one(P["spray"]["tScale"])
        self.fluid = f([d["fuelVec"], d["oxVec"]])
        self.eF, self.eO, self.Ge = one(d["eF"]), one(d["eO"]), one(d["Ge"])
        self.fan = one(25 * math.pi / 180)

    @staticmethod
    def pcg(v):
        m = 0xffffffff
        s = (v * 747796405 + 2891336453) & m
        w = (((s >> ((s >> 28) + 4)) ^ s) * 277803737) & m
        return (w >> 22) ^ w

    def rnd(self, ids, n):
        return (self.pcg((ids + n * 7919) & 0xffffffff) & 0xffffff).double() / 16777216.0

    def wall(self, x, y):
        ex = self.ex
        i, j = torch.floor(x).long(), torch.floor(y).long()
        inside = (i >= 0) & (j >= 0) & (i < ex.Nx) & (j < ex.Nr)
        return inside & ex.solid[0][j.clamp(0, ex.Nr - 1), i.clamp(0, ex.Nx - 1)]

    def step(self, Q, S):
        ex, p = self.ex, self.ex.p
        dt = ex.dt.reshape(())
        num = lambda t: t.reshape(())  # noqa: E731
        a, b = self.PA, self.PB
        idx = torch.arange(RING, device=ex.dev)
        ids = idx ^ ((self.seed * 2654435761) & 0xffffffff)
        spawn = (idx - self.head) % RING < 4
        gi, gj = torch.floor(a[:, 0]).long().clamp(0, ex.Nx - 1), torch.floor(a[:, 1]).long().clamp(0, ex.Nr - 1)
        w = [Q[k][0, gj + 2, gi + 2] for k in range(8)]
        inside = S[0, gj + 2, gi + 2]
        live = b[:, 1] > 0
        fl = self.fluid[(b[:, 2] >= 0.5).long()]
        m, d, dts = b[:, 1], b[:, 0], dt * self.tScale
        rm = ((1 - w[4]) * num(p["gas"][0]) + w[5] * num(p["Rs"][0]) + w[7] * num(p["Rs"][1]) +
              (w[4] - w[5] - w[7]).clamp(min=0) * num(p["Rs"][2]))
        T = w[3] / (w[0] * rm) * num(p["gas"][2])
        rg = w[0] * 1.225
        Ur = torch.sqrt((w[1] - a[:, 2]) ** 2 + (w[2] - a[:, 3]) ** 2) * 287.6 + 1e-3
        mu = 1.458e-6 * T * torch.sqrt(T) / (T + 110.4)
        Re = rg * Ur * d / mu
        tau = 18 * mu * (1 + 0.15 * Re.clamp(max=1000.0) ** 0.687) / (fl[:, 0] * d * d)
        e = torch.exp(-dts * tau)
        vx, vy = w[1] + (a[:, 2] - w[1]) * e, w[2] + (a[:, 3] - w[2]) * e
        cp = rm * 287.05 * (w[6] + 1)
        Bs = (cp * (T - fl[:, 1])).clamp(min=0) / fl[:, 2]
        K = 8 * (mu / 0.7) / fl[:, 0] * torch.log(1 + Bs) * (1 + 0.27 * torch.sqrt(Re))
        d2 = d * d - K * dts
        dn = torch.where(d2 > 1e-12, torch.sqrt(d2.clamp(min=0)), torch.zeros_like(d))
        f = dn / d
        mn = torch.where(dn > 0, m * f * f * f, torch.zeros_like(m))
        we = rg * Ur * Ur * dn / fl[:, 3]
        dst = 12 * fl[:, 3] / (rg * Ur * Ur)
        tb = 3 * dn / Ur * torch.sqrt(fl[:, 0] / rg)
        brk = mix(dn, dst.clamp(min=2e-6), 1 - torch.exp(-dts / tb))
        dn = torch.where((we > 12) & (dn > 0), brk, dn)
        xi = b[:, 3]
        hit = (xi > 0) & (a[:, 0] >= xi)
        sp, phi = torch.sqrt(vx * vx + vy * vy), (self.rnd(ids, 5) - 0.5) * 2 * self.fan
        vx, vy = torch.where(hit, sp * torch.cos(phi), vx), torch.where(hit, sp * torch.sin(phi), vy)
        dn, xi = torch.where(hit, 0.25 * dn, dn), torch.where(hit, torch.zeros_like(xi), xi)
        x, y = a[:, 0] + vx * dt, a[:, 1] + vy * dt
        y, vy = torch.where(y < 0, -y, y), torch.where(y < 0, -vy, vy)
        vx, x = torch.where(x < 0, vx.abs() * 0.3, vx), x.abs()
        inw, hx, hr = self.wall(x, y), self.wall(x, a[:, 1]), self.wall(a[:, 0], y)
        fx, fr = inw & (hx | ~hr), inw & (hr | ~hx)
        x, vx = torch.where(fx, a[:, 0], x), torch.where(fx, -0.3 * vx, vx)
        y, vy = torch.where(fr, a[:, 1], y), torch.where(fr, -0.3 * vy, vy)
        dm = m - mn
        C = torch.stack((dm, mn * (a[:, 2] - vx) + dm * a[:, 2], mn * (a[:, 3] - vy) + dm * a[:, 3]), 1)
        gone = (x >= ex.Nx) | (y >= ex.Nr) | (mn <= 0)
        oA = torch.stack((x, y, vx, vy), 1)
        oB = torch.stack((dn, mn, b[:, 2], xi), 1)
        dead = torch.tensor([-1.0, -1.0, 0.0, 0.0], dtype=torch.float64, device=ex.dev)
        oA, oB = torch.where(gone[:, None], dead, oA), torch.where(gone[:, None], torch.zeros_like(oB), oB)
        walk = torch.stack((a[:, 0] + 1, (a[:, 1] - 0.5).clamp(min=0.05), a[:, 2].clamp(min=0), a[:, 3]), 1)
        oA, oB = torch.where(inside[:, None], walk, oA), torch.where(inside[:, None], b, oB)
        C = torch.where(inside[:, None], torch.zeros_like(C), C)
        oA, oB = torch.where(live[:, None], oA, a), torch.where(live[:, None], oB, b)
        C = torch.where(live[:, None], C, torch.zeros_like(C))
        # births; what an old parcel still carried goes to the gas
        t = (self.rnd(ids, 1) * 255.999).long()
        e1, e2, e3 = (self.tab[k][t] for k in range(3))
        ang = e1[:, 2] + (self.rnd(ids, 2) - 0.5) * 2 * e2[:, 2]
        r = (e1[:, 1] + (self.rnd(ids, 3) - 0.5) * e2[:, 3]).clamp(min=0.05)
        nd = e2[:, 1] * torch.exp((self.rnd(ids, 4) - 0.5) * 1.4)
        nA = torch.stack((e1[:, 0], r, e1[:, 3] * torch.cos(ang), e1[:, 3] * torch.sin(ang)), 1)
        nB = torch.stack((nd, torch.full_like(nd, 1.0) * self.mhat * dt / 4, e2[:, 0], e3[:, 0]), 1)
        old = torch.where(live[:, None], torch.stack((m, m * a[:, 2], m * a[:, 3]), 1), torch.zeros_like(C))
        oA, oB = torch.where(spawn[:, None], nA, oA), torch.where(spawn[:, None], nB, oB)
        C = torch.where(spawn[:, None], old, C)
        # deposits into the group host of the old position's cell, then into the gas
        C = C.masked_fill((a[:, 0] < 0)[:, None], 0.0)
        cell = ex.host[0][gj, gi]
        src = torch.zeros(4, ex.Nr * ex.Nx, dtype=torch.float64, device=ex.dev)
        typ = b[:, 2]
        for k, v in enumerate((C[:, 0] * (1 - typ), C[:, 0] * typ, C[:, 1], C[:, 2])):
            src[k].index_add_(0, cell, v)
        s = src[:, ex.host.reshape(-1)].view(4, 1, ex.Nr, ex.Nx)
        A, B = [ex.at_host(k) for k in ex.A], [ex.at_host(k) for k in ex.B]
        inv = 1 / ex.gV.clamp(min=1e-6)
        dm = s[0] + s[1]
        rho = A[0].clamp(min=RHO_MIN)
        ux, uy = A[1] / rho, A[2] / rho
        rn_ = A[0] + dm * inv
        mx, my = A[1] + s[2] * inv, A[2] + s[3] * inv
        E = A[3] + (s[0] * self.eF + s[1] * self.eO + (ux * s[2] + uy * s[3])) * inv
        G = mix(B[2], self.Ge, (dm * inv / rn_).clamp(max=1.0))
        E = torch.maximum(E, 0.02 * A[3] + 0.5 * rn_ * ((mx / rn_) ** 2 + (my / rn_) ** 2) + P_MIN * G)
        none = (dm == 0) & (s[2] == 0) & (s[3] == 0)
        keep = lambda new, was: torch.where(none, was, new)  # noqa: E731
        ex.A, ex.B = ex.fill_solid([keep(v, w_) for v, w_ in zip((rn_, mx, my, E), A)],
                                   [keep(v, w_) for v, w_ in zip((B[0] + dm * inv, B[1] + s[0] * inv, G,
                                                                  B[3] + s[1] * inv), B)])
        self.PA, self.PB = oA, oB
        self.head, self.seed = (self.head + 4) % RING, (self.seed + 1) & 0xffffffff


def exact(case, seed):
    members = members_of(case, seed)
    groups = {}
    for k, m in enumerate(members):
        groups.setdefault((m[0].Nx, m[0].Nr), []).append(k)
    A, B, info = ([None] * len(members) for _ in range(3))
    spray = None
    for rows in groups.values():
        ex = Exact([members[k] for k in rows])
        if case["config"] == "spray":
            s, P, inj, _, _ = members[0]
            spray = ExactSpray(ex, P, inj, *parcels_of(case, s, P, inj, seed))
        for _ in range(case["steps"]):
            Q, S = ex.step()
            if spray is not None:
                spray.step(Q, S)
        if case["kind"] == "frame":
            return exact_frame(ex, members[0])
        for q, k in enumerate(rows):
            A[k], B[k] = (x[:, q].reshape(4, -1).t() for x in (ex.A, ex.B))
            info[k] = torch.stack([ex.dt[q, 0, 0]] + [ex.t[q, 0, 0]] * 3)
    return outputs_of(torch.cat(A), torch.cat(B), torch.stack(info), spray.PA if spray else None,
                      spray.PB if spray else None, ex.inj)


def exact_frame(ex, member):
    s, P = member[0], member[1]
    q = ex.prims(ex.A, ex.B)
    c = ex.sound(q)
    M = torch.sqrt(q[1] ** 2 + q[2] ** 2) / c
    Rm = ((1 - q[4]) * P["RaN"] + q[5] * P["Rs"][0] + q[7] * P["Rs"][1] +
          (q[4] - q[5] - q[7]).clamp(min=0) * P["Rs"][2])
    T = q[3] / (q[0] * Rm) * physics.T_REF
    scaled = (T - P["Ta"]) / max(s.cfg["Tc"] - P["Ta"], 1.0)
    field = torch.stack((M / 6.0, q[4], scaled, M), -1)
    shut = torch.tensor([0.0, 0.0, 0.0, -1.0], dtype=torch.float64, device=field.device)
    field = torch.where(ex.solid[..., None], shut, field)[0]
    A, B = ex.A[:, 0].permute(1, 2, 0), ex.B[:, 0].permute(1, 2, 0)
    j = torch.as_tensor(np.asarray(s.geo["jWall"]).reshape(-1, 4)[:, 0].astype(np.int64), device=field.device)
    i = torch.arange(s.Nx, device=field.device)
    j = j.clamp(0, s.Nr - 1)
    wall = torch.stack([x[0][j, i] for x in (q[1], q[2], q[3], c)], -1)
    return {"field": field, "dt": ex.dt.reshape(1), "t": ex.t.reshape(1), "A": A[:, s.iExit].reshape(-1),
            "B": B[:, s.iExit].reshape(-1), "probe": A[0, s.iChamber].reshape(-1), "wall": wall.reshape(-1)}
