"""The bounds-checked build on the paths of the device-resident steps: the
cluster kernel and the step graph, uniform and quad meshes, with diffusion and
with cells that are not plain. No check may fire, and the results equal the
default build's bit for bit."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = r'''
import json, sys
import numpy as np
sys.path.insert(0, ROOT)
from mantlepar_b200 import synthetic as sy
from mantlepar_b200.transport import Transport, TransportConfig
out = {}
for nx, ny, quad in ((20, 20, False), (2, 2, False), (31, 33, False), (48, 40, False), (20, 24, True), (3, 2, True), (36, 40, True)):
    for name, diffusion in (("plain", 0.0), ("pure", 1e-3), ("plain", 1e-3)):
        w = sy.Workload(nx=nx, ny=ny, seed=5)
        xy = sy.quad_vertices(w, sy.MESH_PERTURBED, 0.2, seed=11) if quad else None
        t = Transport(w, TransportConfig(cfl=0.4, integrator=3, diffusivity=diffusion), vertices=xy)
        t.set_thermal_bc((1, 2, 0, 1), (0.9, -0.02, 0.0, 0.4))
        t.set_face_velocity(*(sy.face_velocity_quads(w, xy) if quad else sy.face_velocity(w)))
        H, C = sy.initial_state(w)
        t.set_state(H, C if name == "plain" else 0.0 * C)
        code, reps = t.step(6, raise_on_error=False)
        out["%dx%d %s %s %g" % (nx, ny, quad, name, diffusion)] = [[code], list(t.get_time())] + [a.tolist() for a in t.get_state()]
        t.close()
print(json.dumps(out))
'''


def run_cases(checked: bool):
    env = dict(os.environ, MP_CHECKED="1" if checked else "0")
    r = subprocess.run([sys.executable, "-c", "ROOT = %r\n" % ROOT + CASES], capture_output=True, text=True, env=env, cwd=ROOT,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_checked_build_steps_as_the_default_build(cuda_lib):
    from mantlepar_b200 import build
    build.build_checked()
    checked, default = run_cases(True), run_cases(False)
    assert checked.keys() == default.keys()
    for k, values in default.items():
        assert values[0] == [0], k
        for a, b in zip(checked[k], values):
            assert np.array_equal(np.asarray(a), np.asarray(b)), k
