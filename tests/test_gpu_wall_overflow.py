"""A wall temperature so large that the gradient at the wall overflows is
refused, wherever the wall's cells are plain and wherever they are not."""
import numpy as np
import pytest

from mantlepar_b200 import synthetic as sy

pytestmark = pytest.mark.gpu
TYPES, VALUES = (1, 0, 0, 0), (1e308, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("pure", [False, True])
@pytest.mark.parametrize("nx,ny,quad", [(20, 20, False), (48, 40, False), (20, 24, True)])
def test_transport(cuda_lib, nx, ny, quad, pure):
    from mantlepar_b200._capi import MPError
    from mantlepar_b200.transport import Transport, TransportConfig
    w = sy.Workload(nx=nx, ny=ny, seed=5)
    xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
    t = Transport(w, TransportConfig(diffusivity=1e-4), vertices=xy)
    t.set_thermal_bc(TYPES, VALUES)
    t.set_face_velocity(*(sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w)))
    H, C = sy.initial_state(w)
    t.set_state(H, 0.0 * C if pure else C)
    with pytest.raises(MPError) as e:
        t.rhs()
    assert e.value.code == 72
    code, _ = t.step(2, raise_on_error=False)
    assert code == 72
    t.close()


@pytest.mark.parametrize("quad", [False, True])
def test_preheat(cuda_lib, quad):
    from mantlepar_b200.preheat import Preheat, PreheatConfig
    w = sy.Workload(nx=12, ny=10, seed=5)
    xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
    p = Preheat(w, PreheatConfig(end=1.0, cfl=0.5, diffusivity=1e-4, thermal_type=TYPES, thermal_value=VALUES), vertices=xy)
    p.set_velocity((sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w))[0])
    p.set_state(*sy.initial_state(w))
    p.begin()
    code, rows = p.advance(2, raise_on_error=False)
    p.close()
    assert code == 72 and rows == []
