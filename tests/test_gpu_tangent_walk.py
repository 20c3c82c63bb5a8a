"""The differentiable step's force lists: a body's first 128 forces are walked
from shared memory, the others from the list in memory. Values and
derivatives are the tangent oracle's (to test_gpu_tangent's bounds) on both
sides of the line, with manifolds and with springs beyond it.
"""
import importlib

import numpy as np
import pytest

from test_gpu_tangent import check, generic_seeds, run_both

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


@pytest.mark.parametrize("boxes,springs", [(127, 0), (128, 0), (129, 0), (60, 67), (60, 69), (60, 100)])
def test_long_force_lists(abi, scenes, backend_mod, boxes, springs):
    s = scenes.Scene("plate")
    s.params = dict(gravity=-1.0, iterations=2)
    side = int(np.ceil(np.sqrt(boxes)))
    s.box((0.6 * side + 2.0, 0.6 * side + 2.0, 1.0), 500.0, 0.5, (0.0, 0.0, 0.0))
    for k in range(boxes):
        x, y = 0.6 * (k % side - (side - 1) / 2), 0.6 * (k // side - (side - 1) / 2)
        s.box((0.4, 0.4, 0.4), 500.0, 0.5, (x, y, 0.7 - 1e-3 * (1 + k % 5)))
    for k in range(springs):  # from the plate up to boxes far above it
        b = s.box((0.4, 0.4, 0.4), 500.0, 0.5, (0.9 * (k % 10), 0.9 * (k // 10), 6.0))
        s.spring(0, b, (0.1 * (k % 7), 0.0, 0.5), (0.0, 0.0, 0.0), 200.0)
    ref, got, gpu = run_both(abi, backend_mod, s, 2, generic_seeds(abi, s.world()))
    check(ref, got)
    gpu.destroy()
