"""Which failure a preheat step reports when several cells and edges fail."""
import numpy as np
import pytest
import torch

from mantlepar_b200 import synthetic as sy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["advance", "rhs"])
def test_reconstruction_failure_comes_before_the_edges(cuda_lib, call):
    """A state with a NaN in its last cell and backflow through the outflow-only
    bottom wall, on a mesh of several waves of blocks: the reconstruction of the
    first cell whose stencil holds the NaN is reported (a step reconstructs every
    cell before its first flux), whichever block fails first."""
    from mantlepar_b200._capi import MPError
    from mantlepar_b200.preheat import Preheat, PreheatConfig
    nx, ny = 1290, 4536
    w = sy.Workload(nx=nx, ny=ny)
    edges = nx * (ny + 1) + (nx + 1) * ny
    vn = torch.zeros(edges * 5, dtype=torch.float64, device="cuda")
    vn[:5 * nx] = -0.1                       # the bottom wall's outward normal is its canonical one
    H = torch.full((w.cells,), 0.5, dtype=torch.float64, device="cuda")
    C = torch.full_like(H, 0.3)
    H[-1] = float("nan")
    p = Preheat(w, PreheatConfig(end=1.0, dt_initial=1e-3, dt_max=1e-2, cfl=0.5, H_policy=1))
    p.set_velocity(vn)
    p.set_state(H, C)
    p.begin()
    first = (ny - 2) * nx + nx - 2
    if call == "advance":
        code, rows = p.advance(3, raise_on_error=False)
        assert rows == []
        message = p._lib.mp_last_error_string().decode()
    else:
        with pytest.raises(MPError) as e:
            p.rhs()
        code, message = e.value.code, str(e.value)
    p.close()
    assert code == 72 and f"cell {first}:" in message
