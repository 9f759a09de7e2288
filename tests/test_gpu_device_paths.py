"""Device-resident steps on both of their forms, the cluster kernel of small
meshes and the step graph of larger ones: the stream they run on, and their
agreement with the host-driven loop."""
import numpy as np
import pytest
import torch

from mantlepar_b200 import synthetic as sy

pytestmark = pytest.mark.gpu


def transport(nx, ny, cfg, quad=False, stream=None, seed=5):
    from mantlepar_b200.transport import Transport
    w = sy.Workload(nx=nx, ny=ny, seed=seed)
    xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
    t = Transport(w, cfg, stream=stream, vertices=xy)
    t.set_face_velocity(*(sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w)))
    t.set_state(*sy.initial_state(w))
    return t


@pytest.mark.parametrize("nx,ny,quad", [(20, 20, False), (48, 40, False), (20, 24, True), (36, 40, True)])
def test_steps_run_on_the_handles_stream(cuda_lib, nx, ny, quad):
    """Steps of a handle on a stream of its own neither wait for the default
    stream nor run there: with that stream busy throughout, they finish, and
    give the states and reports of the host-driven loop."""
    from mantlepar_b200.transport import TransportConfig
    cfg = TransportConfig(cfl=0.4, integrator=3)
    side = torch.cuda.Stream()
    got = []
    for device in (True, False):
        t = transport(nx, ny, cfg, quad, side.cuda_stream)
        t.set_device_steps(device)
        reps = t.step(2)[1]                  # allocations and the graph's capture
        torch.cuda.synchronize()
        torch.cuda._sleep(2_000_000_000)     # about one second of the default stream
        busy = torch.cuda.Event()
        busy.record()
        reps += t.step(70)[1]
        assert not busy.query()
        got.append((reps, t.get_time(), t.get_state()))
        torch.cuda.synchronize()
        t.close()
    assert got[0][:2] == got[1][:2]
    for x, y in zip(got[0][2], got[1][2]):
        assert np.array_equal(x, y)


def untidy_state(w, kind):
    """States whose cells are not plain: pure component, eutectic composition,
    or a band of C = 0 beside a ramp."""
    n = np.arange(w.cells)
    x, y = (n % w.nx + 0.5) / w.nx, (n // w.nx + 0.5) / w.ny
    H = 0.05 + 0.6 * y + 0.02 * sy.unit_noise(w.seed, 0, n.astype(np.uint64))
    C = {"pure": 0.0 * x, "eutectic": 0.5 + 0.0 * x, "ramp": 0.3 * np.clip(x - 0.4, 0.0, 1.0)}[kind]
    return H, C


@pytest.mark.parametrize("kind", ["pure", "eutectic", "ramp"])
@pytest.mark.parametrize("nx,ny,quad", [(9, 7, False), (25, 33, False), (48, 40, False), (9, 7, True), (19, 25, True),
                                        (36, 40, True)])
def test_cells_that_are_not_plain_agree_on_every_path(cuda_lib, nx, ny, quad, kind):
    """The tested forms of the cell phase, faces and diffusion are compiled
    into the stage kernels, the batch's kernels and the cluster kernel: device
    steps, the host-driven loop and a batch give the same doubles."""
    from mantlepar_b200.batch import Batch
    from mantlepar_b200.transport import Transport, TransportConfig
    w = sy.Workload(nx=nx, ny=ny, seed=5)
    xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
    cfg = TransportConfig(cfl=0.4, integrator=3, diffusivity=1e-3)
    types, values = (1, 2, 0, 1), (0.9, -0.02, 0.0, 0.4)
    velocity = sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w)
    state = untidy_state(w, kind)
    got = []
    for device in (True, False):
        t = Transport(w, cfg, vertices=xy)
        t.set_device_steps(device)
        t.set_thermal_bc(types, values)
        t.set_face_velocity(*velocity)
        t.set_state(*state)
        code, reps = t.step(5, raise_on_error=False)
        got.append((code, reps, t.get_time(), t.get_state()))
        t.close()
    b = Batch([w] if not quad else [sy.Workload(nx=4, ny=4)], cfg)
    k = b.add_quads(w, xy) if quad else 0
    b.set_thermal_bc(types, values)
    if quad:
        b.set_face_velocity(0, *sy.face_velocity(sy.Workload(nx=4, ny=4)))
        b.set_state(0, *sy.initial_state(sy.Workload(nx=4, ny=4)))
    b.set_face_velocity(k, *velocity)
    b.set_state(k, *state)
    b.step(5)
    s = b.get_state(k)
    b.close()
    a, h = got
    assert a[:3] == h[:3]
    for x, y in zip(a[3], h[3]):
        assert np.array_equal(x, y)
    if kind != "ramp":
        assert a[0] == 0
    if a[0] == 0:
        assert s["status"] == 0
        for x, name in zip(a[3], ("H", "C", "T", "phi")):
            assert np.array_equal(x, s[name]), name


@pytest.mark.parametrize("nx,ny,quad,diffusion,lithostatic", [
    (32, 48, False, 0.0, False), (32, 32, False, 1e-3, False), (25, 41, False, 1e-3, False), (32, 32, False, 0.0, True),
    (25, 41, False, 0.0, True), (32, 32, True, 0.0, False), (20, 32, True, 1e-3, False), (27, 24, True, 1e-3, False)])
def test_both_sides_of_the_cluster_kernels_limits(cuda_lib, nx, ny, quad, diffusion, lithostatic):
    """Meshes at the limits of the cluster kernel (1536 cells, 1024 with
    diffusion or a lithostatic pressure; quads 1024 and 640) and just beyond:
    the host-driven loop's states and reports."""
    from mantlepar_b200.transport import TransportConfig
    cfg = TransportConfig(cfl=0.4, integrator=3, diffusivity=diffusion)
    got = []
    for device in (True, False):
        t = transport(nx, ny, cfg, quad)
        t.set_device_steps(device)
        if diffusion:
            t.set_thermal_bc((1, 2, 0, 1), (0.9, -0.02, 0.0, 0.4))
        if lithostatic:
            t.set_pressure_model(t.LITHOSTATIC, 1.1)
        code, reps = t.step(5)
        got.append((code, reps, t.get_time(), t.get_state()))
        t.close()
    assert got[0][:3] == got[1][:3]
    for x, y in zip(got[0][3], got[1][3]):
        assert np.array_equal(x, y)
