"""The first pack of a process loads the unit of the solve kernels, and of them
those that its steps can launch: it takes no more than five times a later one
(2 to 3 measured; 7 to 11 with a compressed image), for a scene of each kind."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = """
import importlib, sys, time
abi = importlib.import_module("avbd-sandbox_gb300.abi")
scenes = importlib.import_module("avbd-sandbox_gb300.scene")
backend = importlib.import_module("avbd-sandbox_gb300.backend")
s = getattr(scenes, sys.argv[1])()
gpu = backend.GpuBackend(abi.default_params(**s.params, contact_model=int(sys.argv[2])))
w = s.world()
t = []
for _ in range(9):
    t0 = time.perf_counter()
    gpu.pack(w)
    t.append(time.perf_counter() - t0)
gpu.step(2)
gpu.idle()
print(t[0] / sorted(t[1:])[4])
"""


@pytest.mark.parametrize("scene", ["cube_stack", "brick_wall", "heavy_chain"])
@pytest.mark.parametrize("model", [0, 1])
def test_first_pack(scene, model):
    ratios = []
    for _ in range(3):  # (the host may be busy with something else)
        out = subprocess.run([sys.executable, "-c", PROGRAM, scene, str(model)], cwd=ROOT, capture_output=True, text=True,
                             timeout=300)
        assert out.returncode == 0, out.stderr[-2000:]
        ratios.append(float(out.stdout.split()[-1]))
        if ratios[-1] < 5.0:
            return
    assert min(ratios) < 5.0, ratios
