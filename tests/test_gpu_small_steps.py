"""Scenes of fewer than 1,024 bodies build their adjacency in one block: pairs,
manifolds, colouring and the stepped positions are the oracle's on both sides
of the line.
"""
import importlib

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu
POS_TOL = 1e-5  # the FP32 single-step bound of the parity tests


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


@pytest.mark.parametrize("bodies", [1, 2, 33, 1023, 1024, 1025])
def test_one_block_and_many(abi, scenes, backend_mod, bodies):
    s = scenes.Scene("rows")
    for k in range(bodies):  # columns of four on a grid, the lowest of each fixed
        x, y, z = k // 4 % 24, k // 96, k % 4
        s.box((1.0, 1.0, 1.0), 0.0 if z == 0 else 500.0, 0.5, (1.2 * x, 1.2 * y, 0.995 * z))
    params = abi.default_params(gravity=-9.81, iterations=4, body_order=abi.ORDER_PRIORITY)
    gpu = backend_mod.GpuBackend(params)
    gpu.pack(s.world())
    o = Oracle(params, s.world())
    gpu.step(1)
    o.step(1)
    gpu.idle()
    out, ref = gpu.read_state(manifolds=True), o.state()
    for a, b in zip(gpu.read_pairs(), o.pairs()):
        assert np.array_equal(a, b)
    assert out.manifold_dict() == ref.manifold_dict() and (bodies == 1 or out.m_count > bodies // 2 - 1)
    (gc, gn), (oc, on) = gpu.read_coloring(), o.coloring()
    assert gn == on and np.array_equal(gc, oc)
    assert np.abs(out.pos - ref.pos).max() < POS_TOL
    gpu.destroy()
