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


def failing_minimum(nx, ny, cfg_of, quad):
    """A minimum step for which a run gives up at its first retry, after a
    stage of the rejected attempt was evaluated; and that step's index."""
    t = transport(nx, ny, cfg_of(1e-14), quad)
    reps = t.step(200)[1]
    t.close()
    k = next(i for i, r in enumerate(reps) if r["retries"])
    attempted = reps[k]["dt"] * 2 ** reps[k]["retries"]
    assert all(r["dt"] > 0.75 * attempted for r in reps[:k])
    return 0.75 * attempted, k


@pytest.mark.parametrize("integrator", [2, 3])
@pytest.mark.parametrize("nx,ny,quad", [(20, 20, False), (48, 40, False), (20, 24, True), (36, 40, True)])
def test_state_after_a_step_that_fails_in_a_stage(cuda_lib, nx, ny, quad, integrator):
    """A step given up after a stage was evaluated leaves that stage's T and
    phi, as the host-driven loop does: single mesh and batch."""
    from mantlepar_b200.batch import Batch
    from mantlepar_b200.transport import TransportConfig

    def cfg(dt_min):
        return TransportConfig(cfl=0.4, integrator=integrator, dt_min=dt_min)

    dt_min, k = failing_minimum(nx, ny, cfg, quad)
    got = []
    for device in (True, False):
        t = transport(nx, ny, cfg(dt_min), quad)
        t.set_device_steps(device)
        if k:
            t.step(k)
        accepted = t.get_state()
        code, reps = t.step(70, raise_on_error=False)
        assert code == 91
        state = t.get_state()
        assert np.array_equal(state[0], accepted[0]) and not np.array_equal(state[2], accepted[2])
        got.append((reps, t.get_time(), state))
        t.close()
    assert got[0][:2] == got[1][:2]
    for x, y in zip(got[0][2], got[1][2]):
        assert np.array_equal(x, y)

    # The same mesh in a batch, beside one that runs on.
    w, other = sy.Workload(nx=nx, ny=ny, seed=5), sy.Workload(nx=4, ny=3)
    states = []
    for device in (True, False):
        b = Batch([other], cfg(dt_min))
        b.set_device_steps(device)
        xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
        i = b.add_quads(w, xy) if quad else b.add(w)
        b.set_face_velocity(0, *sy.face_velocity(other))
        b.set_state(0, *sy.initial_state(other))
        b.set_face_velocity(i, *(sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w)))
        b.set_state(i, *sy.initial_state(w))
        reps = b.step(k + 3)
        s = b.get_state(i)
        assert s["status"] == 91
        states.append((reps, s))
        b.close()
    assert states[0][0] == states[1][0]
    for name in ("H", "C", "T", "phi"):
        assert np.array_equal(states[0][1][name], states[1][1][name]), name
    for x, name in zip(got[0][2], ("H", "C", "T", "phi")):
        assert np.array_equal(x, states[0][1][name]), name


FORMS = [(20, 20, False), (48, 40, False), (20, 24, True), (36, 40, True)]


def run_both(make, steps):
    got = []
    for device in (True, False):
        t = make(device)
        code, reps = t.step(steps, raise_on_error=False)
        got.append(dict(code=code, reps=reps, time=t.get_time(), state=t.get_state(), syncs=t.host_syncs(),
                        message=t._lib.mp_last_error_string() if code else b""))
        t.close()
    a, b = got
    for key in ("code", "reps", "time", "message"):
        assert a[key] == b[key], key
    for x, y in zip(a["state"], b["state"]):
        assert np.array_equal(x, y)
    return a, b


@pytest.mark.parametrize("integrator", [2, 3])
@pytest.mark.parametrize("nx,ny,quad", FORMS)
def test_long_runs_with_retries(cuda_lib, nx, ny, quad, integrator):
    """Several chunks of 64 steps with CFL retries among them."""
    from mantlepar_b200.transport import TransportConfig

    def make(device):
        t = transport(nx, ny, TransportConfig(cfl=0.4, integrator=integrator), quad)
        t.set_device_steps(device)
        return t

    a, b = run_both(make, 200)
    assert a["code"] == 0 and sum(r["retries"] for r in a["reps"]) > 0
    assert a["syncs"] <= 1 + 4 and b["syncs"] >= 3 * 200


@pytest.mark.parametrize("nx,ny,quad", FORMS)
@pytest.mark.parametrize("control", ["end", "fixed", "fixed too large", "minimum", "setters"])
def test_time_controls_and_setters(cuda_lib, nx, ny, quad, control):
    """An end time inside the run, the fixed control below and above the CFL
    bound, a minimum step that no attempt meets, and setters between runs."""
    from mantlepar_b200.transport import Transport, TransportConfig
    options = {"fixed": dict(dt_initial=2e-5), "fixed too large": dict(dt_initial=1.0), "minimum": dict(dt_min=10.0),
               "setters": dict(diffusivity=1e-4)}.get(control, {})

    def make(device):
        t = transport(nx, ny, TransportConfig(cfl=0.4, integrator=3, **options), quad)
        t.set_device_steps(device)
        if control == "end":
            dt = t.step(3)[1][-1]["dt"]
            t.set_time_control(Transport.CFL, t.get_time()[0] + 10.5 * dt)
        elif control.startswith("fixed"):
            t.set_time_control(Transport.FIXED)
        elif control == "setters":
            t.step(10)
            t.set_thermal_bc((1, 1, 0, 0), (0.9, 0.2, 0.0, 0.0))
            t.step(10)
            t.set_state(*sy.initial_state(sy.Workload(nx=nx, ny=ny, seed=9)))
        return t

    a, _ = run_both(make, 20)
    assert a["code"] == {"fixed too large": 63, "minimum": 91}.get(control, 0)
    if control == "end":
        assert a["reps"][-1]["dt"] == 0.0


def test_a_batch_counts_the_launches_of_its_graph(cuda_lib):
    """A batch of one mesh runs the kernels of the single mesh's step graph:
    the same launches for the same steps and attempts."""
    from mantlepar_b200._capi import kernel_launches
    from mantlepar_b200.batch import Batch
    from mantlepar_b200.transport import TransportConfig
    cfg = TransportConfig(cfl=0.4, integrator=3)
    w = sy.Workload(nx=48, ny=40, seed=5)
    t, b = transport(48, 40, cfg), Batch([w], cfg)
    b.set_face_velocity(0, *sy.face_velocity(w))
    b.set_state(0, *sy.initial_state(w))
    counts = []
    for x in (t, b):
        x.step(2)
        before = kernel_launches()
        x.step(60)
        counts.append(kernel_launches() - before)
        x.close()
    assert counts[0] == counts[1]
