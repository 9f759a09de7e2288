"""A state so rough that the sum of a cell's unnormalised weights is subnormal
(its reciprocal overflows) is refused: 2x2 cells have one candidate each, whose
weight (epsilon A / (sigma + epsilon A))^5 is about 1e-318 at 1e30."""
import numpy as np
import pytest

from mantlepar_b200 import synthetic as sy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("scale,refused", [(1e30, True), (1e28, False)])
def test_subnormal_weights(cuda_lib, scale, refused, quad):
    from mantlepar_b200._capi import MPError
    from mantlepar_b200.preheat import Preheat, PreheatConfig
    w = sy.Workload(nx=2, ny=2)
    xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, 11) if quad else None
    p = Preheat(w, PreheatConfig(end=1.0, cfl=0.5), vertices=xy)
    p.set_velocity((sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w))[0])
    p.set_state(np.array([1.0, 2.0, 3.0, 1.5]) * scale, np.full(4, 0.3))
    p.begin()
    if refused:
        with pytest.raises(MPError) as e:
            p.rhs()
        assert e.value.code == 72
    else:
        assert np.all(np.isfinite(p.rhs()[0]))
    p.close()
