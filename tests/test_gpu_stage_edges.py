"""The stage kernels at the sizes and data where their fast forms meet their
general ones: tile edges and remainders of the 32x4-cell blocks, meshes
without an interior cell, and a domain so small that the smoothness
indicators leave the range of the product form of the weights. Oracle: the
restated CPU driver on the same inputs.

Tolerances. Per-cell |x - ref| / max(|ref|, 1e-3 max|ref|). Limiter factors
1e-11: a factor is a ratio of differences of averages, and two roundings of
the stencil tables move the worst of 3.3 million such cells by 1e-11. Stage
T 1e-12, RHS 1e-12 of its largest value (the bars of the golden stages)."""
from __future__ import annotations

import numpy as np
import pytest

from mantlepar_b200 import synthetic as sy

pytestmark = pytest.mark.gpu


def per_cell(x, ref):
    x, ref = np.asarray(x).reshape(-1), np.asarray(ref).reshape(-1)
    return np.max(np.abs(x - ref) / np.maximum(np.abs(ref), 1e-3 * np.max(np.abs(ref))))


def pair(w, **config):
    """The GPU instance and the oracle's with the same inputs."""
    from mantlepar_b200.transport import Transport, TransportConfig
    from oracle import pyoracle as po
    o = po.TransportOracle(sy.material_s(), w, lib=po.restated(), integrator=w.integrator, **config)
    t = Transport(w, TransportConfig(cfl=w.cfl, integrator=w.integrator, **config))
    H, C = sy.initial_state(w)
    vs, ud = sy.face_velocity(w)
    for x in (o, t):
        x.set_face_velocity(vs, ud)
        x.set_state(H, C)
    return t, o


@pytest.mark.parametrize("scale", [1.0, 1e-6])
@pytest.mark.parametrize("nx,ny", [(2, 2), (2, 7), (3, 3), (31, 4), (33, 5), (65, 9)])
def test_reconstruction_and_limiter(nx, ny, scale):
    # scale 1e-6: epsilon * area is 1e-12 smaller, sigma / (epsilon * area) up
    # to 1e15, beyond the product form of the weights.
    w = sy.Workload(nx=nx, ny=ny, x1=0.5 * scale, y1=scale, seed=nx + ny, noise_H=0.05 * scale if scale < 1 else 0.05)
    if scale < 1:
        # Keep the enthalpy of the unit domain: 1 - y needs its own height.
        H = (1.0 - (np.arange(nx * ny) // nx + 0.5) / ny) + 0.05 * sy.unit_noise(w.seed, 0, np.arange(nx * ny, dtype=np.uint64))
        C = sy.initial_state(w)[1]
    t, o = pair(w)
    if scale < 1:
        t.set_state(H, C)
        o.set_state(H, C)
    code, *factors = o.limiter()
    assert code == 0
    for g, r in zip(t.limiter(), factors):
        assert np.max(np.abs(g - r)) <= 1e-11
    got, (code, ref) = t.rhs(), o.rhs()
    assert code == 0
    assert per_cell(got["T"], ref["T"]) <= 1e-12
    for k in ("rhsH", "rhsC"):
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * np.max(np.abs(ref[k]))


def patchy_state(w):
    """Columns of pure component (C = 0), of eutectic composition (C = Xe) and
    ordinary ones, two-solid to solid + liquid: cells that take the tested
    phase evaluation beside cells that do not need it, and the edges between."""
    i = np.arange(w.cells) % w.nx
    band = (3 * i) // w.nx
    C = np.where(band == 0, 0.0, np.where(band == 1, 0.3 + 0.02 * sy.unit_noise(w.seed, 1, np.arange(w.cells, dtype=np.uint64)), 0.5))
    H = 0.05 + 0.6 * (np.arange(w.cells) // w.nx + 0.5) / w.ny + 0.03 * sy.unit_noise(w.seed, 0, np.arange(w.cells, dtype=np.uint64))
    return H, C


@pytest.mark.parametrize("config", [{}, {"theta": 2.0}, {"lf_global": 1, "lf_global_speed": 1.0}, {"C_policy": 2}, {"H_policy": 2}],
                         ids=["plain", "darcy_exponent", "global_lf", "zero_flux_C", "zero_flux_H"])
@pytest.mark.parametrize("nx,ny", [(4, 3), (37, 11)])
def test_faces_of_mixed_cells_and_walls(nx, ny, config):
    w = sy.Workload(nx=nx, ny=ny, seed=7)
    t, o = pair(w, inflow_H=0.6, inflow_C=0.31, **config)
    H, C = patchy_state(w)
    vs, ud = sy.face_velocity(w)
    vs = vs.copy()
    vs[: nx * (ny + 1)] += 0.05            # through-flow: inflow at one wall, outflow at the other
    for x in (t, o):
        x.set_state(H, C)
        x.set_face_velocity(vs, ud)
    got, (code, ref) = t.rhs(), o.rhs()
    assert code == 0
    assert per_cell(got["T"], ref["T"]) <= 1e-12
    assert per_cell(got["phi"], ref["phi"]) <= 1e-12
    for k in ("rhsH", "rhsC", "rate"):
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * np.max(np.abs(ref[k]))


@pytest.mark.parametrize("family", [1, 2], ids=["perturbed", "stretched"])
@pytest.mark.parametrize("config", [{}, {"theta": 2.0}, {"lf_global": 1, "lf_global_speed": 1.0}, {"H_policy": 2}],
                         ids=["plain", "darcy_exponent", "global_lf", "zero_flux_H"])
@pytest.mark.parametrize("nx,ny", [(2, 3), (35, 9)])
def test_quad_mesh_of_mixed_cells_and_walls(nx, ny, config, family):
    from mantlepar_b200.transport import Transport, TransportConfig
    from oracle import pyoracle as po
    w = sy.Workload(nx=nx, ny=ny, seed=7)
    bc = dict(inflow_H=0.6, inflow_C=0.31, **config)
    o = po.TransportOracle(sy.material_s(), w, lib=po.restated(), integrator=3, mesh_family=family, perturbation=0.2,
                           mesh_seed=11, **bc)
    xy = o.vertices()
    t = Transport(w, TransportConfig(cfl=w.cfl, integrator=3, **bc), vertices=xy)
    vs, ud = sy.face_velocity_quads(w, xy)
    vs = vs + 0.05 * (ud / w.darcy)
    H, C = patchy_state(w)
    for x in (t, o):
        x.set_state(H, C)
        x.set_face_velocity(vs, ud)
    got, (code, ref) = t.rhs(), o.rhs()
    assert code == 0
    assert per_cell(got["T"], ref["T"]) <= 1e-12
    assert per_cell(got["phi"], ref["phi"]) <= 1e-12
    for k in ("rhsH", "rhsC", "rate"):
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * np.max(np.abs(ref[k]))
    code, *factors = o.limiter()
    assert code == 0
    for g, r in zip(t.limiter(), factors):
        assert np.max(np.abs(g - r)) <= 1e-11


@pytest.mark.parametrize("types,values", [((1, 2, 0, 1), (0.9, -0.02, 0.0, 0.4)), ((1, 1, 1, 1), (0.9, 0.2, 0.5, 0.5)),
                                          ((2, 0, 1, 2), (0.01, 0.0, 0.6, -0.03))], ids=["mixed", "temperature", "flux"])
@pytest.mark.parametrize("nx,ny,patchy", [(2, 2, False), (33, 6, False), (37, 11, True)])
def test_diffusion_and_source(nx, ny, patchy, types, values):
    # Diffusion with every kind of wall, lithostatic pressure and the
    # adiabatic source, whose cell velocities a warp stages 32 cells at a
    # time (66 and 407 cells: last warps of 2 and 23 cells).
    import dataclasses
    from mantlepar_b200.transport import Transport, TransportConfig
    from oracle import pyoracle as po
    w = sy.Workload(nx=nx, ny=ny, seed=5)
    mat = dataclasses.replace(sy.material_s(), rho=100.0, alpha0=3e-5)
    o = po.TransportOracle(mat, w, lib=po.restated(), integrator=2, theta=2.0)
    t = Transport(w, TransportConfig(material=mat, cfl=w.cfl, integrator=2, theta=2.0, diffusivity=0.02))
    assert o.set_diffusion(0.02, types, values) == 0
    t.set_thermal_bc(types, values)
    assert o.set_pressure_model(1, 1.1) in (0, None)
    t.set_pressure_model(t.LITHOSTATIC, 1.1)
    H, C = patchy_state(w) if patchy else sy.initial_state(w)
    vs, ud = sy.face_velocity(w)
    for x in (t, o):
        x.set_cell_velocity(*sy.cell_velocity(w))
        x.set_face_velocity(vs, ud)
        x.set_state(H, C)
    got, (code, ref) = t.rhs(), o.rhs()
    assert code == 0
    assert per_cell(got["T"], ref["T"]) <= 1e-12
    assert per_cell(got["phi"], ref["phi"]) <= 1e-12
    for k in ("rhsH", "rhsC", "rate"):
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * np.max(np.abs(ref[k]))


@pytest.mark.parametrize("mesh", ["uniform", "lithostatic", "perturbed"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (9, 3), (16, 16), (17, 31), (32, 32), (31, 33), (32, 48), (41, 38)])
def test_small_meshes_step_as_the_host_loop(nx, ny, mesh):
    # Steps in one cluster kernel (up to 1536 cells, quads 1024) and in the
    # graph beyond, both against the host-driven loop: bit for bit, with
    # plain and other cells, retries and an end time inside the run.
    from mantlepar_b200.transport import Transport, TransportConfig
    w = sy.Workload(nx=nx, ny=ny, seed=nx)
    xy = sy.quad_vertices(w, 1, 0.2, 11) if mesh == "perturbed" else None
    vs, ud = sy.face_velocity(w) if xy is None else sy.face_velocity_quads(w, xy)
    H, C = patchy_state(w) if nx > 8 else sy.initial_state(w)
    got = []
    for device in (True, False):
        t = Transport(w, TransportConfig(cfl=0.4, integrator=3 if nx % 2 else 2), vertices=xy)
        t.set_device_steps(device)
        if mesh == "lithostatic":
            t.set_pressure_model(t.LITHOSTATIC, 1.02)
        t.set_face_velocity(vs, ud)
        t.set_state(H, C)
        code, reps = t.step(3, raise_on_error=False)
        if code == 0:
            t.set_time_control(t.CFL, reps[-1]["time"] + 1.5 * reps[-1]["dt"])
            code, more = t.step(4, raise_on_error=False)
            reps += more
        got.append((code, reps, t.get_time(), t.get_state()))
        t.close()
    a, b = got
    assert a[:3] == b[:3]
    for x, y in zip(a[3], b[3]):
        assert np.array_equal(x, y)
