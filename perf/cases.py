"""Performance cases of the library's public entry points on one GPU.

A case is a dict of plain values. `listed()` names the fixed ones, `draw()`
gives more of the same ranges, `prepare()` makes what a user's program holds
before the call (device inputs from a seed, the handle), `run()` is one pass
through the entry points, `work()` the bytes and operations the pass cannot do
without, and `exact()` the same outputs from plain 64-bit torch arithmetic.

The workloads are the repository's own: uniform nx x ny meshes on
[0, 0.5] x [0, 1] with the streamfunction flow, perturbed and sine-stretched
quad meshes, batches of uneven meshes, the legacy preheat and the phase
equilibrium on its own. All data is FP64, the only type the library computes in.

Kinds
  phase    EutecticModel.evaluate_batch on device arrays (pointwise equilibrium)
  steps    Transport: load a state, advance SSP Runge-Kutta steps, read H, C, T, phi
           ("velocity": the flow supplier's face velocities are loaded as well,
           as a coupled program does before every step)
  batch    Batch: the same for many meshes of different size advanced together
  preheat  Preheat: forward-Euler steps of a running integration, read H
           ("diagnostics": and the cell averages of T and phi)
"""
import itertools
import math

import numpy as np
import torch

from mantlepar_b200 import synthetic as sy
from mantlepar_b200._capi import check
from mantlepar_b200.batch import Batch
from mantlepar_b200.phase import EutecticModel
from mantlepar_b200.preheat import Preheat, PreheatConfig
from mantlepar_b200.transport import Transport, TransportConfig

F64 = torch.float64
DOMAIN = (0.0, 0.5, 0.0, 1.0)
CFL = 0.4
KAPPA = 1e-4                                   # thermal diffusivity of the product features and the preheat
WALL_TYPES, WALL_VALUES = (1, 1, 0, 0), (0.9, 0.2, 0.0, 0.0)   # walls bottom, top, left, right
SURFACE_Y = 1.1                                # lithostatic pressure: height of the surface
THROUGH = 0.05                                 # upward through-flow of the preheat
PREHEAT_DT = 1e-4
PHASE_FIELDS = ["phi1", "phi2", "phil", "cl", "cs", "TDp", "Tep", "dTD_dCD", "dTD_dHD", "region", "flags"]


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # Pointwise equilibrium of a few points: a line plot, one mesh row. Call latency.
        {"name": "phase_1000", "kind": "phase", "n": 1000, "pressure": "array", "fields": "all"},
        # Post-processing of a whole large field at one pressure. Memory-bound.
        {"name": "phase_4m", "kind": "phase", "n": 4000037, "pressure": "constant", "fields": "all"},
        # The smallest product run (20x20 grid), SSPRK3: the length of a step is latency.
        {"name": "steps_20x20", "kind": "steps", "mesh": "uniform", "nx": 20, "ny": 20, "field": "noise",
         "integrator": 3, "steps": 10, "theta": 0.0, "features": "plain", "velocity": False},
        # One step of a coupled run on an odd mesh: new face velocities, one SSPRK2 step, results out.
        {"name": "coupled_61x127", "kind": "steps", "mesh": "uniform", "nx": 61, "ny": 127, "field": "smooth",
         "integrator": 2, "steps": 1, "theta": 2.0, "features": "plain", "velocity": True},
        # An ordinary mid-size run with ragged edges.
        {"name": "steps_321x643", "kind": "steps", "mesh": "uniform", "nx": 321, "ny": 643, "field": "noise",
         "integrator": 3, "steps": 2, "theta": 0.0, "features": "plain", "velocity": False},
        # The headline mesh.
        {"name": "steps_1280x2560", "kind": "steps", "mesh": "uniform", "nx": 1280, "ny": 2560, "field": "noise",
         "integrator": 3, "steps": 2, "theta": 0.0, "features": "plain", "velocity": False},
        # The product input's physics: diffusion with wall temperatures, lithostatic pressure, adiabatic source.
        {"name": "product_256x512", "kind": "steps", "mesh": "uniform", "nx": 256, "ny": 512, "field": "smooth",
         "integrator": 2, "steps": 2, "theta": 0.0, "features": "product", "velocity": False},
        # A small perturbed-quadrilateral mesh (per-cell tables), latency.
        {"name": "quads_40x80", "kind": "steps", "mesh": "perturbed", "nx": 40, "ny": 80, "field": "smooth",
         "integrator": 3, "steps": 4, "theta": 0.0, "features": "plain", "velocity": False},
        # A large perturbed-quadrilateral mesh (per-cell tables), throughput.
        {"name": "quads_640x1280", "kind": "steps", "mesh": "perturbed", "nx": 640, "ny": 1280, "field": "noise",
         "integrator": 3, "steps": 1, "theta": 0.0, "features": "plain", "velocity": False},
        # A parameter study: uneven meshes in one batch.
        {"name": "batch_24_uneven", "kind": "batch", "count": 24, "nx_max": 400, "ny_max": 600, "field": "noise",
         "integrator": 3, "steps": 2},
        # The preheat phase of a run on the headline mesh, an output interval of 16 steps.
        {"name": "preheat_1280x2560", "kind": "preheat", "mesh": "uniform", "nx": 1280, "ny": 2560, "field": "smooth",
         "steps": 16, "diagnostics": False},
        # The preheat on a small quad mesh with the final diagnostics.
        {"name": "preheat_quads_101x203", "kind": "preheat", "mesh": "perturbed", "nx": 101, "ny": 203,
         "field": "smooth", "steps": 64, "diagnostics": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh_size(rng, nx_max):
    nx = _log_int(rng, 10, nx_max)
    return nx, max(8, int(nx * rng.uniform(0.8, 2.0)))


def draw(rng):
    kind = rng.choice(["phase", "steps", "steps", "product", "quads", "batch", "preheat"])
    if kind == "phase":
        return {"kind": "phase", "n": _log_int(rng, 1000, 4000000), "pressure": rng.choice(["array", "constant"]),
                "fields": rng.choice(["all", "T_phi"])}
    field = rng.choice(["noise", "smooth"])
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 64), "nx_max": rng.randint(40, 250),
                "ny_max": rng.randint(40, 400), "field": field, "integrator": rng.choice([2, 3]), "steps": 2}
    if kind == "preheat":
        nx, ny = _mesh_size(rng, 1280)
        mesh = rng.choice(["uniform", "perturbed", "stretched"])
        if mesh != "uniform":
            nx, ny = max(10, nx // 3), max(8, ny // 3)
        return {"kind": "preheat", "mesh": mesh, "nx": nx, "ny": ny, "field": field, "steps": rng.randint(4, 16),
                "diagnostics": rng.random() < 0.3 and nx < 300}
    case = {"kind": "steps", "field": field, "integrator": rng.choice([2, 3]), "steps": rng.randint(1, 3),
            "theta": rng.choice([0.0, 0.0, 2.0]), "features": "product" if kind == "product" else "plain",
            "velocity": rng.random() < 0.3, "mesh": rng.choice(["perturbed", "stretched"]) if kind == "quads" else "uniform"}
    case["nx"], case["ny"] = _mesh_size(rng, {"steps": 1000, "product": 500, "quads": 400}[kind])
    return case


# ----------------------------------------------------------------- the inputs

def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(seed % (1 << 62))


def _vertices(mesh, nx, ny, seed):
    """(ny+1, nx+1, 2) vertex array: uniform, interior vertices displaced by up to 0.2 of the spacing, or x and y
    stretched by a sine."""
    dev = _device()
    x0, x1, y0, y1 = DOMAIN
    s = torch.arange(nx + 1, dtype=F64, device=dev) / nx
    t = torch.arange(ny + 1, dtype=F64, device=dev) / ny
    if mesh == "stretched":
        s, t = torch.sin(0.5 * math.pi * s), torch.sin(0.5 * math.pi * t)
    x = (x0 + (x1 - x0) * s)[None, :].expand(ny + 1, nx + 1)
    y = (y0 + (y1 - y0) * t)[:, None].expand(ny + 1, nx + 1)
    V = torch.stack([x, y], -1).clone()
    if mesh == "perturbed":
        u = torch.rand(ny - 1, nx - 1, 2, dtype=F64, device=dev, generator=_generator(seed + 7))
        h = torch.tensor([(x1 - x0) / nx, (y1 - y0) / ny], dtype=F64, device=dev)
        V[1:-1, 1:-1] += 0.2 * h * (2.0 * u - 1.0)
    return V


def _flow(x, y, amp):
    """Solid velocity of the streamfunction amp sin(2 pi x) sin(pi y)."""
    return (math.pi * amp * torch.sin(2 * math.pi * x) * torch.cos(math.pi * y),
            -2 * math.pi * amp * torch.cos(2 * math.pi * x) * torch.sin(math.pi * y))


GP = torch.tensor(np.polynomial.legendre.leggauss(5)[0])
GW = torch.tensor(np.polynomial.legendre.leggauss(5)[1])


def _face_velocity(V, amp, through=0.0):
    """Normal solid and Darcy (0, 0.01) velocities at the 5 Gauss points of every edge, edges along i first; the
    streamfunction part is zero on the walls."""
    t = (0.5 * (1.0 + GP)).to(V.device)
    vs_all, ud_all = [], []
    for a, b, axis in ((V[:, :-1], V[:, 1:], 0), (V[:-1], V[1:], 1)):
        d = b - a
        n = torch.stack([d[..., 1], -d[..., 0]], -1) / torch.hypot(d[..., 0], d[..., 1])[..., None]
        p = a[..., None, :] + t[:, None] * d[..., None, :]
        vx, vy = _flow(p[..., 0], p[..., 1], amp)
        vs = vx * n[..., None, 0] + vy * n[..., None, 1]
        vs.select(axis, 0).zero_()
        vs.select(axis, -1).zero_()
        vs += through * n[..., None, 1]
        vs_all.append(vs.reshape(-1, 5))
        ud_all.append((0.01 * n[..., None, 1]).expand_as(vs).reshape(-1, 5))
    return torch.cat(vs_all).contiguous(), torch.cat(ud_all).contiguous()


def _corners(V):
    return V[:-1, :-1], V[:-1, 1:], V[1:, 1:], V[1:, :-1]


def _lerp(r, a, b):
    return 0.5 * (1.0 - r) * a + 0.5 * (1.0 + r) * b


def _bilinear(r, s, c):
    return _lerp(s, _lerp(r, c[0], c[1]), _lerp(r, c[3], c[2]))


def _cell_velocity(V, amp):
    """Vertical solid and Darcy velocities at the 25 cell points, [cell, b*5 + a]."""
    c = _corners(V)
    vy = torch.stack([_flow(*_bilinear(float(a), float(b), c).unbind(-1), amp)[1] for b in GP for a in GP], -1)
    return vy.reshape(-1).contiguous(), torch.full((vy.numel(),), 0.01, dtype=F64, device=V.device)


def _state(field, V, g):
    """Cell averages H, C: the seeded noise of the benchmark workloads, or a smooth state as it is some way into a run."""
    c = _corners(V)
    x, y = (0.25 * (c[0] + c[1] + c[2] + c[3])).unbind(-1)
    if field == "noise":
        H = (1.0 - y) + 0.05 * torch.rand(y.shape, dtype=F64, device=V.device, generator=g)
        return H.reshape(-1), (0.3 + 0.02 * torch.rand(y.shape, dtype=F64, device=V.device, generator=g)).reshape(-1)
    r = torch.rand(4, dtype=F64, device=V.device, generator=g)
    H = (1.0 - y) + 0.03 + 0.02 * torch.sin(4 * math.pi * x + 6 * r[0]) * torch.cos(3 * math.pi * y + 6 * r[1])
    C = 0.31 + 0.01 * torch.cos(6 * math.pi * x + 6 * r[2]) * torch.sin(2 * math.pi * y + 6 * r[3])
    return H.reshape(-1).contiguous(), C.reshape(-1).contiguous()


def _amplitude(g):
    return 0.05 + 0.1 * float(torch.rand(1, dtype=F64, device=_device(), generator=g))


def _material(features):
    m = sy.material_s()
    if features == "product":
        m.rho, m.alpha0 = 100.0, 3e-5
    return m


def _mesh_inputs(case, seed):
    g = _generator(seed)
    V = _vertices(case["mesh"], case["nx"], case["ny"], seed)
    amp = _amplitude(g)
    H, C = _state(case["field"], V, g)
    return V, amp, H, C


def _phase_inputs(case, seed):
    g, n = _generator(seed), case["n"]
    r = torch.rand(4, n, dtype=F64, device=_device(), generator=g)
    Xe = sy.material_s().Xe
    H, C = 1.6 * r[0], 0.98 * Xe * r[1]
    C[r[2] < 0.02] = 0.0                       # some points of the pure component
    P = 2e8 * r[3]
    return H.contiguous(), C.contiguous(), P.contiguous()


def _batch_meshes(case, seed):
    rng = np.random.default_rng(1000 + case["count"] + case["nx_max"])   # the study's meshes: fixed by the case
    size = lambda top: max(20, int(round(math.exp(rng.uniform(math.log(20), math.log(top))))))  # noqa: E731
    out = []
    for k in range(case["count"]):
        nx, ny = size(case["nx_max"]), size(case["ny_max"])
        out.append((nx, ny) + _mesh_inputs(dict(case, mesh="uniform", nx=nx, ny=ny), seed + 101 * k))
    return out


def prepare(case, seed):
    s = dict(case)
    if case["kind"] == "phase":
        H, C, P = _phase_inputs(case, seed)
        s.update(model=EutecticModel(sy.material_s()), H=H, C=C, P=P if case["pressure"] == "array" else None,
                 fields_wanted=PHASE_FIELDS if case["fields"] == "all" else ["TDp", "phil"])
        return s
    if case["kind"] == "batch":
        meshes = _batch_meshes(case, seed)
        b = Batch([sy.Workload(nx=nx, ny=ny) for nx, ny, *_ in meshes], TransportConfig(cfl=CFL, integrator=case["integrator"]))
        for i, (_, _, V, amp, _, _) in enumerate(meshes):
            b.set_face_velocity(i, *_face_velocity(V, amp))
        s.update(batch=b, states=[(H, C) for *_, H, C in meshes], out=[torch.empty(4, H.numel(), dtype=F64, device=H.device) for *_, H, _ in meshes])
        return s
    V, amp, H, C = _mesh_inputs(case, seed)
    w = sy.Workload(nx=case["nx"], ny=case["ny"])
    xy = None if case["mesh"] == "uniform" else V.reshape(-1).cpu().numpy()
    if case["kind"] == "preheat":
        p = Preheat(w, PreheatConfig(end=1e9, max_steps=1 << 40, dt_initial=PREHEAT_DT, dt_max=PREHEAT_DT, cfl=0.5,
                                     diffusivity=KAPPA, thermal_type=WALL_TYPES, thermal_value=WALL_VALUES), vertices=xy)
        p.set_velocity(_face_velocity(V, amp, THROUGH)[0])
        p.set_state(H, C)
        p.begin()
        s.update(preheat=p, H=torch.empty_like(H))
        return s
    product = case["features"] == "product"
    t = Transport(w, TransportConfig(material=_material(case["features"]), cfl=CFL, integrator=case["integrator"],
                                     theta=case["theta"], diffusivity=KAPPA if product else 0.0), vertices=xy)
    if product:
        t.set_thermal_bc(WALL_TYPES, WALL_VALUES)
        t.set_pressure_model(t.LITHOSTATIC, SURFACE_Y)
        t.set_cell_velocity(*_cell_velocity(V, amp))
    vs, ud = _face_velocity(V, amp)
    t.set_face_velocity(vs, ud)
    s.update(transport=t, H=H, C=C, vs=vs, ud=ud, out=torch.empty(4, H.numel(), dtype=F64, device=H.device))
    return s


# ------------------------------------------------------------------- one pass

def run(s):
    if s["kind"] == "phase":
        out, _, _ = s["model"].evaluate_batch(s["H"], s["C"], s["P"], 1e8, fields=s["fields_wanted"])
        return out
    if s["kind"] == "batch":
        b = s["batch"]
        for i, (H, C) in enumerate(s["states"]):
            b.set_state(i, H, C)
        b.step(s["steps"])
        for i, o in enumerate(s["out"]):      # the C entry point takes device pointers; Batch.get_state copies to the host
            check(b._lib.mp_batch_get_state(b._h, i, o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), o[3].data_ptr(),
                                            None, None, None))
        return s["out"]
    if s["kind"] == "preheat":
        s["preheat"].advance(s["steps"])
        s["preheat"].get_state_into(s["H"])
        return [s["H"], *s["preheat"].diagnostics()] if s["diagnostics"] else [s["H"]]
    t, o = s["transport"], s["out"]
    if s["velocity"]:
        t.set_face_velocity(s["vs"], s["ud"])
    t.set_state(s["H"], s["C"])
    t.step(s["steps"])
    t.get_state_into(o[0], o[1], o[2], o[3])
    return o


def work(case):
    """Bytes: each input read and each output written once per evaluation. Per cell and stage of the transport 224 B
    (stage state and U^n in, next state out, 2 owned edges x 5 points x 2 velocities in, T and phi out), on a quad mesh
    also its 184 table entries; per cell and preheat step 96 B (H in and out, 2 edges x 5 velocities). Operations: the
    reconstruction, limiter, phase quadrature and face fluxes as the scheme states them."""
    if case["kind"] == "phase":
        n = case["n"]
        ins = 24 if case["pressure"] == "array" else 16
        return {"bytes": n * (ins + (74 if case["fields"] == "all" else 16)), "flops": 60.0 * n}
    if case["kind"] == "batch":
        rng = np.random.default_rng(1000 + case["count"] + case["nx_max"])
        size = lambda top: max(20, int(round(math.exp(rng.uniform(math.log(20), math.log(top))))))  # noqa: E731
        cells = sum(size(case["nx_max"]) * size(case["ny_max"]) for _ in range(case["count"]))
        stages = 1 + case["integrator"] * case["steps"]
        return {"bytes": cells * 224.0 * stages, "flops": cells * 4000.0 * stages}
    cells = float(case["nx"] * case["ny"])
    tables = 0 if case["mesh"] == "uniform" else 184 * 8
    if case["kind"] == "preheat":
        return {"bytes": cells * case["steps"] * (96 + tables), "flops": cells * case["steps"] * 600.0}
    stages = 1 + case["integrator"] * case["steps"]
    product = case["features"] == "product"
    return {"bytes": cells * stages * (224 + tables + (400 if product else 0)),
            "flops": cells * stages * (6500.0 if product else 4000.0)}


# --------------------------------------------------- the same in plain torch

def _derived(m):
    dT = m.Tm0 - m.Te0
    return {"dT": dT, "LD": m.L / (m.cp * dT), "TDe0": m.Te0 / dT, "l0": math.sqrt(m.mus * m.k0 / m.mul)}


def _phase(m, H, C, Tep):
    """Equilibrium at (H, C) with eutectic temperature Tep: dict of fields."""
    LD, Xe = _derived(m)["LD"], m.Xe
    Tep = torch.as_tensor(Tep, dtype=F64, device=H.device).expand_as(H)
    Tmp, r = Tep + 1.0, C / Xe
    Heut, Hliq = Tep + LD * r, Tep + (1.0 - r) + LD
    pure = C == 0.0
    a = H - Tmp
    disc = torch.hypot(a, 2.0 * torch.sqrt(LD * r))
    melt = torch.where(a >= 0, (a + disc) / (2 * LD), 2 * r / (disc - a))
    emelt = torch.minimum(r, (H - Tep) / LD)
    esecond = (C - emelt * Xe).clamp(min=0.0)
    one, zero = torch.ones_like(H), torch.zeros_like(H)
    solid = [~pure & (H <= Tep), pure & (H <= Tmp)]
    liquid = H >= Hliq
    eut = ~pure & ~solid[0] & ~liquid & (H <= Heut)
    melting = pure & ~solid[1] & ~liquid
    mix = ~pure & ~solid[0] & ~liquid & ~eut
    liquid = liquid & ~solid[0] & ~solid[1]

    def pick(**v):
        out = zero
        for k, mask in (("two", solid[0]), ("ps", solid[1]), ("eut", eut), ("pm", melting), ("mix", mix), ("liq", liquid)):
            if k in v:
                out = torch.where(mask, v[k], out)
        return out
    phil = pick(eut=emelt, pm=a / LD, mix=melt, liq=one).clamp(0.0, 1.0)
    phi2 = pick(two=C, eut=esecond).clamp(0.0, 1.0)
    phi1 = pick(two=1.0 - C, ps=one, eut=1.0 - emelt - esecond, pm=1.0 - a / LD, mix=1.0 - melt).clamp(0.0, 1.0)
    cl = pick(eut=Xe * one, mix=C / melt, liq=C)
    cl = torch.where(phil > 0, cl, zero)
    sol = phi1 + phi2
    cs = torch.where(sol > 0, phi2 / sol, zero)
    T = pick(two=H, ps=H, eut=Tep, pm=Tmp, mix=torch.where(a >= 0, Tmp - r / melt, H - LD * melt), liq=H - LD)
    dH = pick(two=one, ps=one, mix=torch.where(a >= 0, 2 * LD / disc * (r / (disc + a)), 0.5 * (1 - a / disc)), liq=one)
    dC = pick(mix=-(LD / disc) / Xe)
    dC = torch.where(pure & (H > Tep) & ~liquid, -(LD / a.abs()) / Xe, dC)
    return {"phi1": phi1, "phi2": phi2, "phil": phil, "cl": cl, "cs": cs, "TDp": T, "Tep": Tep, "dTD_dCD": dC, "dTD_dHD": dH}


def _binomial_shift(p, S, dx, dy):
    """Coefficients of p(x + dx, y + dy), monomial j*S + i of x^i y^j."""
    out = []
    for jn in range(S):
        for i_n in range(S):
            out.append(sum(p[..., j * S + i] * (math.comb(i, i_n) * math.comb(j, jn)) * dx ** (i - i_n) * dy ** (j - jn)
                           for j in range(jn, S) for i in range(i_n, S)))
    return torch.stack(out, -1)


def _value(D, x, y):
    r = [D[..., 3 * j] + x * (D[..., 3 * j + 1] + x * D[..., 3 * j + 2]) for j in range(3)]
    return r[0] + y * (r[1] + y * r[2])


def _derivative(p, S, x, y, dx, dy):
    return sum(math.perm(i, dx) * math.perm(j, dy) * p[..., j * S + i] * x ** (i - dx) * y ** (j - dy)
               for j in range(dy, S) for i in range(dx, S))


G3, W3 = (v.tolist() for v in np.polynomial.legendre.leggauss(3))


def _jacobian(r, s, c):
    u, v = 0.5 * (1.0 + r), 0.5 * (1.0 + s)
    ex, et = 0.5 * ((1 - v) * (c[1] - c[0]) + v * (c[2] - c[3])), 0.5 * ((1 - u) * (c[3] - c[0]) + u * (c[2] - c[1]))
    return ex[..., 0] * et[..., 1] - ex[..., 1] * et[..., 0]


class _Scheme:
    """The finite-volume scheme on one logically rectangular mesh: ML-WENO(3,2), limiter, phase, Lax-Friedrichs fluxes.
    On a uniform mesh the stencil matrices are those of one cell."""

    def __init__(self, V, uniform, m):
        self.m, self.d, self.V = m, _derived(m), V
        ny, nx = V.shape[0] - 1, V.shape[1] - 1
        self.ny, self.nx, dev = ny, nx, V.device
        self.c = _corners(V)
        self.centre = 0.25 * (self.c[0] + self.c[1] + self.c[2] + self.c[3])
        self.area = 4.0 * _jacobian(0.0, 0.0, self.c)
        self.h = torch.sqrt(self.area)
        ii, jj = torch.arange(nx, device=dev), torch.arange(ny, device=dev)
        self.nbr = lambda A, di, dj: A[(jj + dj).clamp(0, ny - 1)][:, (ii + di).clamp(0, nx - 1)]
        ones = torch.ones(ny, nx, dtype=torch.bool, device=dev)
        inside = {0: ones, -1: (ii > 0)[None, :] & ones, 1: (ii < nx - 1)[None, :] & ones}
        up = {0: ones, -1: (jj > 0)[:, None] & ones, 1: (jj < ny - 1)[:, None] & ones}
        self.stencils = []       # (mask, cell offsets, size, inverse moments, centre shift, smoothness rule)
        x0, x1, y0, y1 = DOMAIN
        for S, oi, oj in ((3, -1, -1), (2, 0, -1), (2, 0, 0), (2, -1, -1), (2, -1, 0)):
            offs = [(oi + i, oj + j) for j in range(S) for i in range(S)]
            mask = inside[oi] & inside[oi + S - 1] & up[oj] & up[oj + S - 1]
            if uniform:
                dx, dy = (x1 - x0) / nx, (y1 - y0) / ny
                q = lambda i, j: [torch.tensor([[[(i + a) * dx, (j + b) * dy]]], dtype=F64, device=dev)  # noqa: E731
                                  for a, b in ((0, 0), (1, 0), (1, 1), (0, 1))]
                quads, target = [q(i, j) for i, j in offs], q(0, 0)
                h, mk = self.h[:1, :1], torch.ones(1, 1, dtype=torch.bool, device=dev)
                h = torch.full_like(h, math.sqrt(dx * dy))
            else:
                quads, target = [[self.nbr(v, i, j) for v in self.c] for i, j in offs], self.c
                h, mk = self.h, mask
            o = 0.25 * (quads[0][0] + quads[S - 1][1] + quads[-1][2] + quads[(S - 1) * S][3])
            loc = [[(v - o) / h[..., None] for v in qd] for qd in quads]
            M = torch.stack([self._moments(qd, S) for qd in loc], -2)
            M = torch.where(mk[..., None, None], M, torch.eye(S * S, dtype=F64, device=dev))
            shift = (0.25 * (target[0] + target[1] + target[2] + target[3]) - o) / h[..., None]
            if S == 3:           # smoothness over the unit reference square of the stencil frame
                rule = [(0.5 * a, 0.5 * b, 0.25 * wa * wb) for b, wb in zip(G3, W3) for a, wa in zip(G3, W3)]
            else:                # over the target cell
                tq = [(v - o) / h[..., None] for v in target]
                A = 4.0 * _jacobian(0.0, 0.0, tq)
                rule = [(*_bilinear(a, b, tq).unbind(-1), wa * wb * _jacobian(a, b, tq) / A)
                        for b, wb in zip(G3, W3) for a, wa in zip(G3, W3)]
            self.stencils.append((mask, offs, S, torch.linalg.inv(M), shift, rule))
        self._edges()

    @staticmethod
    def _moments(c, S):
        total, out = 0.0, [0.0] * (S * S)
        for b, wb in zip(G3, W3):
            for a, wa in zip(G3, W3):
                x, y = _bilinear(a, b, c).unbind(-1)
                w = wa * wb * _jacobian(a, b, c)
                total = total + w
                for j in range(S):
                    for i in range(S):
                        out[j * S + i] = out[j * S + i] + w * x ** i * y ** j
        return torch.stack([v / total for v in out], -1)

    def _edges(self):
        """Per cell and edge (bottom, right, top, left): end points, length, outward normal, Gauss points, and the
        spacing of the samples on the normal lines."""
        c, n2 = self.c, {}
        self.edge = []
        for e in range(4):
            a, b = c[e], c[(e + 1) % 4]
            d = b - a
            ln = torch.hypot(d[..., 0], d[..., 1])
            nrm = torch.stack([d[..., 1], -d[..., 0]], -1) / ln[..., None]
            pts = [_lerp(float(g), a, b) for g in GP]
            for q, p in enumerate(pts):
                best = torch.full_like(ln, math.inf)
                for f in range(4):
                    if f == e:
                        continue
                    t, r = c[(f + 1) % 4] - c[f], p - c[f]
                    ins = t[..., 0] * r[..., 1] - t[..., 1] * r[..., 0]
                    rate = -(t[..., 0] * nrm[..., 1] - t[..., 1] * nrm[..., 0])
                    best = torch.where(rate < 0, torch.minimum(best, ins / -rate), best)
                n2[e, q] = best
            self.edge.append((ln, nrm, pts))
        self.spacing = {}
        ones = torch.ones_like(self.area, dtype=torch.bool)
        self.wall = [ones.clone() for _ in range(4)]
        for e, (di, dj) in enumerate(((0, -1), (1, 0), (0, 1), (-1, 0))):
            w = torch.zeros_like(ones)
            (w[0] if e == 0 else w[:, -1] if e == 1 else w[-1] if e == 2 else w[:, 0]).fill_(True)
            self.wall[e] = w
            for q in range(5):
                other = self.nbr(n2[(e + 2) % 4, 4 - q], di, dj)
                self.spacing[e, q] = torch.where(w, 0.9 * n2[e, q] / 4, 0.9 * torch.minimum(n2[e, q], other) * (2.0 / 3.0))

    def local(self, p, at=()):
        return ((p[..., 0] - self.centre[at][..., 0]) / self.h[at], (p[..., 1] - self.centre[at][..., 1]) / self.h[at])

    def reconstruct(self, u):
        """Deviation polynomials (ny, nx, 9) in the cells' frames."""
        eA = 1e-2 * self.area
        polys, alphas = [], []
        for mask, offs, S, inv, shift, rule in self.stencils:
            d = torch.stack([self.nbr(u, i, j) - u for i, j in offs], -1)
            p = (inv @ d[..., None])[..., 0]
            order = S - 1
            sig = sum(w * sum(_derivative(p, S, x, y, dx, dy) ** 2 for dy in range(S) for dx in range(S) if 0 < dx + dy <= order)
                      for x, y, w in rule)
            r = eA / (sig.clamp(min=0.0) + eA)
            # (sigma + eA)^-7 and ^-5 with eA^-7 divided out.
            alphas.append(torch.where(mask, r ** 7 if S == 3 else eA * eA * r ** 5, torch.zeros_like(r)))
            s = _binomial_shift(p, S, shift[..., 0], shift[..., 1])
            if S == 2:
                z = torch.zeros_like(s[..., 0])
                s = torch.stack([s[..., 0], s[..., 1], z, s[..., 2], s[..., 3], z, z, z, z], -1)
            polys.append(s)
        # Without the order-2 stencil the order-1 weights share another common factor, which cancels here.
        total = sum(alphas)
        return sum((a / total)[..., None] * s for a, s in zip(alphas, polys))

    def samples(self, e, q):
        """Points of the normal-line samples of edge e, point q, on this cell's side: (mask, point)."""
        p, n, sp, wall = self.edge[e][2][q], self.edge[e][1], self.spacing[e, q], self.wall[e]
        for k in range(4):
            d = torch.where(wall, float(k - 4) * sp, (k - 1.5) * sp)
            yield wall | (k < 2), p + d[..., None] * n

    def limit(self, u, D, top):
        lo = hi = u
        for di, dj in itertools.product((-1, 0, 1), (-1, 0, 1)):
            v = self.nbr(u, di, dj)
            lo, hi = torch.minimum(lo, v), torch.maximum(hi, v)
        lo, hi = lo.clamp(min=0.0), hi.clamp(max=top)
        mx = mn = D[..., 0]
        pts = [(None, _bilinear(float(a), float(b), self.c)) for a in GP for b in GP]
        pts += [(None, p) for e in range(4) for p in self.edge[e][2]]
        for mask, p in itertools.chain(pts, *(self.samples(e, q) for e in range(4) for q in range(5))):
            v = _value(D, *self.local(p))
            v = v if mask is None else torch.where(mask, v, D[..., 0])
            mx, mn = torch.maximum(mx, v), torch.minimum(mn, v)
        th = torch.ones_like(u)
        vmax, vmin = u + mx, u + mn
        th = torch.where(vmax > hi, torch.minimum(th, (hi - u) / (vmax - u)), th)
        th = torch.where(vmin < lo, torch.minimum(th, (lo - u) / (vmin - u)), th)
        return torch.where(th < 1.0, (th * (1 - 1e-13)).clamp(min=0.0), th)


class _Transport(_Scheme):
    def __init__(self, V, uniform, features, theta, vs, ud, amp):
        super().__init__(V, uniform, _material(features))
        self.product, self.theta = features == "product", theta
        self.kappa = KAPPA if self.product else 0.0
        nI = self.nx * (self.ny + 1)
        cut = lambda v: (v[:nI].reshape(self.ny + 1, self.nx, 5), v[nI:].reshape(self.ny, self.nx + 1, 5))  # noqa: E731
        self.vs, self.ud = cut(vs), cut(ud)
        if self.product:
            self.cell_v = [v.reshape(self.ny, self.nx, 25) for v in _cell_velocity(V, amp)]
            self.cooling = self.m.alpha0 * self.d["l0"] * self.m.g / self.m.cp

    def tep(self, y):
        if not self.product:
            return self.d["TDe0"]
        return self.d["TDe0"] + self.m.rho * self.m.g * self.d["l0"] / self.m.nu / self.d["dT"] * (SURFACE_Y - y)

    def factor(self, phi):
        return torch.where(phi == 0.0, phi, phi if self.theta == 0.0 else phi ** (1.0 + self.theta))

    def at(self, p, sel):
        x, y = self.local(p, sel)
        return self.u[0][sel] + _value(self.D[0][sel], x, y), self.u[1][sel] + _value(self.D[1][sel], x, y)

    def face(self, L, e, R, wall, vs, ud, sgn):
        """Fluxes H, C, mixture-independent rate of a set of edges: left cells' edge e, right cells R or None."""
        ln, nrm, pts = self.edge[e][0][L], self.edge[e][1][L], [p[L] for p in self.edge[e][2]]
        LD, Xe = self.d["LD"], self.m.Xe
        FH = FC = rate = 0.0
        for q in range(5):
            k = q if sgn > 0 else 4 - q
            s, u = sgn * vs[..., k], sgn * ud[..., k]
            p = pts[q]
            tep = self.tep(p[..., 1])
            hL, cL = self.at(p, L)
            A = _phase(self.m, hL, cL, tep)
            cR, B = cL, A
            wet = self.wet[L]
            if R is not None:
                hR, cR = self.at(p, R)
                B = _phase(self.m, hR, cR, tep)
                wet = wet & self.wet[R]
            cl, cs = 0.5 * (A["cl"] + B["cl"]), 0.5 * (A["cs"] + B["cs"])
            S = A["phil"] + B["phil"]
            phi = torch.where(wet & (S > 0), 2 * A["phil"] * B["phil"] / S, torch.zeros_like(S))
            bulk = phi * cl + (1 - phi) * cs
            clb = torch.where(wet & (S > 0) & (bulk > 0), cl / bulk, torch.zeros_like(S))
            fl = self.factor(phi) * u
            vn, ve = s + fl, s + clb * fl
            if R is not None:
                fh = 0.5 * (vn * (A["TDp"] + B["TDp"]) - vn.abs() * (B["TDp"] - A["TDp"])) - LD * (1 - phi) * s
                fc = 0.5 * (ve * (cL + cR) - ve.abs() * (cR - cL))
            else:                # reservoir H = 1, C = 0.3 where the flow enters
                inC = torch.where(ve < 0, torch.full_like(cL, 0.3), cL)
                Tb = torch.where(vn < 0, _phase(self.m, torch.ones_like(cL), inC, tep)["TDp"], A["TDp"])
                fh = torch.where(vn == 0, torch.zeros_like(vn), vn * Tb - LD * (1 - phi) * s)
                fc = torch.where(ve == 0, torch.zeros_like(ve), ve * inC)
            w = 0.5 * ln * float(GW[q])
            sens = 1.0 + torch.maximum(A["dTD_dCD"].abs(), B["dTD_dCD"].abs())
            FH, FC = FH + w * fh, FC + w * fc
            rate = rate + w * (ve.abs() + vn.abs() + 2 * s.abs()) * sens
            if self.kappa and not (R is None and WALL_TYPES[wall] == 0):
                sp = self.spacing[e, q][L]
                cf = (0.25, -4 / 3, 3.0, -4.0, 25 / 12) if R is None else (1 / 24, -9 / 8, 9 / 8, -1 / 24)
                grad = 0.0
                for k4 in range(4):
                    x = p + ((k4 - 4.0 if R is None else k4 - 1.5) * sp)[..., None] * nrm
                    h, c = self.at(x, L if R is None or k4 < 2 else R)
                    grad = grad + cf[k4] * _phase(self.m, h, c, self.tep(x[..., 1]))["TDp"]
                if R is None:
                    grad = grad + cf[4] * WALL_VALUES[wall]
                FH = FH - w * self.kappa * grad / sp
                rate = rate + w * self.kappa / sp * sum(abs(v) for v in cf[:4])
        return FH, FC, rate

    def rhs(self, H, C):
        """(dH/dt, dC/dt, largest rate, cell averages of T and phi)."""
        self.u = (H, C)
        self.D = []
        for u, top in ((H, math.inf), (C, self.m.Xe)):
            D = self.reconstruct(u)
            self.D.append(D * self.limit(u, D, top)[..., None])
        T = phi = src = src_rate = 0.0
        self.wet = torch.zeros_like(H, dtype=torch.bool)
        for b in range(5):
            for a in range(5):
                p = _bilinear(float(GP[a]), float(GP[b]), self.c)
                P = _phase(self.m, *self.at(p, ()), self.tep(p[..., 1]))
                w = float(GW[a] * GW[b]) * _jacobian(float(GP[a]), float(GP[b]), self.c) / self.area
                T, phi = T + w * P["TDp"], phi + w * P["phil"]
                self.wet |= P["phil"] > 0
                if self.product:
                    v = self.cell_v[0][..., b * 5 + a] + self.factor(P["phil"]) * self.cell_v[1][..., b * 5 + a]
                    src, src_rate = src - w * self.cooling * P["TDp"] * v, src_rate + w * self.cooling * v.abs()
        out = [torch.zeros_like(H) for _ in range(3)]
        full = slice(None)
        for L, e, R, wall, o, es, sgn in (
                ((slice(1, None), full), 0, (slice(None, -1), full), 0, 0, (slice(1, -1), full), 1.0),
                ((slice(0, 1), full), 0, None, 0, 0, (slice(0, 1), full), 1.0),
                ((slice(-1, None), full), 2, None, 1, 0, (slice(-1, None), full), -1.0),
                ((full, slice(None, -1)), 1, (full, slice(1, None)), 2, 1, (full, slice(1, -1)), 1.0),
                ((full, slice(0, 1)), 3, None, 2, 1, (full, slice(0, 1)), -1.0),
                ((full, slice(-1, None)), 1, None, 3, 1, (full, slice(-1, None)), 1.0)):
            F = self.face(L, e, R, wall, self.vs[o][es], self.ud[o][es], sgn)
            for k in range(3):
                out[k][L] += F[k] if k == 2 else -F[k]
                if R is not None:
                    out[k][R] += F[k]
        rH, rC, rate = (v / self.area for v in out)
        return rH + src, rC, float((rate + src_rate).max()), T, phi

    def advance(self, H, C, steps, integrator):
        """Accepted SSP Runge-Kutta steps with the CFL and admissibility retries: H, C, T, phi."""
        ok = lambda h, c: bool((h.min() >= 0) & (c.min() >= 0) & (c.max() <= self.m.Xe) & torch.isfinite(h).all() & torch.isfinite(c).all())  # noqa: E731
        combos = ((0.75, 0.25), (1 / 3, 2 / 3)) if integrator == 3 else ((0.5, 0.5),)
        L = self.rhs(H, C)
        for _ in range(steps):
            dt = CFL / L[2]
            while True:
                h, c, top = H + dt * L[0], C + dt * L[1], L[2]
                good = ok(h, c)
                for a0, a1 in combos:
                    if good:
                        s = self.rhs(h, c)
                        h, c = a0 * H + a1 * (h + dt * s[0]), a0 * C + a1 * (c + dt * s[1])
                        top = max(top, s[2])
                        good = dt * top <= CFL * (1 + 1e-12) and ok(h, c)
                if good:
                    break
                dt *= 0.5
            H, C = h, c
            L = self.rhs(H, C)
        return [v.reshape(-1) for v in (H, C, L[3], L[4])]


def _preheat(case, V, amp, H, C):
    s = _Scheme(V, case["mesh"] == "uniform", sy.material_s())
    nI, H, C = s.nx * (s.ny + 1), H.reshape(s.ny, s.nx), C.reshape(s.ny, s.nx)
    vn = _face_velocity(V, amp, THROUGH)[0]
    vn = (vn[:nI].reshape(s.ny + 1, s.nx, 5), vn[nI:].reshape(s.ny, s.nx + 1, 5))
    full = slice(None)
    groups = (((slice(1, None), full), 0, (slice(None, -1), full), 0, 0, (slice(1, -1), full), 1.0),
              ((slice(0, 1), full), 0, None, 0, 0, (slice(0, 1), full), 1.0),
              ((slice(-1, None), full), 2, None, 1, 0, (slice(-1, None), full), -1.0),
              ((full, slice(None, -1)), 1, (full, slice(1, None)), 2, 1, (full, slice(1, -1)), 1.0),
              ((full, slice(0, 1)), 3, None, 2, 1, (full, slice(0, 1)), -1.0),
              ((full, slice(-1, None)), 1, None, 3, 1, (full, slice(-1, None)), 1.0))
    inner, outer = 1 / 24 - 9 / 8, 1 / 4 - 4 / 3 + 3 - 4   # sums of the derivative weights of one side's samples

    def evaluate(H, rate_only=False):
        D = None if rate_only else s.reconstruct(H)
        out = torch.zeros_like(H)
        for L, e, R, wall, o, es, sgn in groups:
            F = 0.0
            for q in range(5):
                v = sgn * vn[o][es][..., q if sgn > 0 else 4 - q]
                w = 0.5 * s.edge[e][0][L] * float(GW[q])
                conduct = w * KAPPA / s.spacing[e, q][L] * abs(inner if R is not None else outer)
                if R is None and WALL_TYPES[wall] == 0:
                    conduct = 0.0
                if rate_only:
                    F = F + w * v.abs() + conduct
                    continue
                p = s.edge[e][2][q][L]
                uL = H[L] + _value(D[L], *s.local(p, L))
                if R is not None:
                    uR = H[R] + _value(D[R], *s.local(p, R))
                    F = F + w * 0.5 * (v * (uL + uR) - v.abs() * (uR - uL)) + conduct * (H[L] - H[R])
                else:
                    F = F + w * v * torch.where(v < 0, torch.ones_like(uL), uL) + conduct * (H[L] - WALL_VALUES[wall])
            out[L] += F if rate_only else -F
            if R is not None:
                out[R] += F
        return out / s.area

    dt = min(PREHEAT_DT, 0.5 / float(evaluate(H, rate_only=True).max()))
    for _ in range(case["steps"]):
        H = H + dt * evaluate(H)
    if not case["diagnostics"]:
        return [H.reshape(-1)]
    T = phi = 0.0
    DH, DC = s.reconstruct(H), s.reconstruct(C)
    for b in range(5):
        for a in range(5):
            p = _bilinear(float(GP[a]), float(GP[b]), s.c)
            x, y = s.local(p)
            P = _phase(s.m, H + _value(DH, x, y), C + _value(DC, x, y), s.d["TDe0"])
            w = float(GW[a] * GW[b]) * _jacobian(float(GP[a]), float(GP[b]), s.c) / s.area
            T, phi = T + w * P["TDp"], phi + w * P["phil"]
    return [H.reshape(-1), T.reshape(-1), phi.reshape(-1)]


def exact(case, seed):
    if case["kind"] == "phase":
        H, C, P = _phase_inputs(case, seed)
        m = sy.material_s()
        d = _derived(m)
        P = P if case["pressure"] == "array" else torch.full_like(P, 1e8)
        out = _phase(m, H, C, d["TDe0"] + P / m.nu / d["dT"])
        wanted = PHASE_FIELDS if case["fields"] == "all" else ["TDp", "phil"]
        return {f: out.get(f) for f in wanted}   # region and flags are whole numbers
    if case["kind"] == "batch":
        got = []
        for nx, ny, V, amp, H, C in _batch_meshes(case, seed):
            t = _Transport(V, True, "plain", 0.0, *_face_velocity(V, amp), amp)
            got.append(torch.stack(t.advance(H.reshape(ny, nx), C.reshape(ny, nx), case["steps"], case["integrator"])))
        return got
    V, amp, H, C = _mesh_inputs(case, seed)
    if case["kind"] == "preheat":
        return _preheat(case, V, amp, H, C)
    t = _Transport(V, case["mesh"] == "uniform", case["features"], case["theta"], *_face_velocity(V, amp), amp)
    return torch.stack(t.advance(H.reshape(case["ny"], case["nx"]), C.reshape(case["ny"], case["nx"]), case["steps"], case["integrator"]))
