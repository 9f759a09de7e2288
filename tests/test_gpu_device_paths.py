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
