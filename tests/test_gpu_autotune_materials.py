"""The autotuner puts every contact's restitution bias back with the rest of the
state: the next step reads it to tell a new impact from one under way."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def test_biases_are_put_back(abi, scenes, backend_mod):
    s, mat = scenes.material_scene("drop")
    w = s.world()
    w.set_materials(**mat)
    gpu = backend_mod.GpuBackend(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY,
                                                    contact_model=abi.CONTACT_MATERIALS))
    gpu.pack(w)
    for _ in range(60):  # until an impact is under way
        gpu.step(1)
        gpu.idle()
        before = gpu.read_state(manifolds=True)
        if np.any(before.m_restitution_bias[:before.m_count] > 0):
            break
    assert np.any(before.m_restitution_bias[:before.m_count] > 0)
    gpu.autotune(3)
    after = gpu.read_state(manifolds=True)
    gpu.destroy()
    m = before.m_count
    assert after.m_count == m
    for f in ("body_a", "body_b", "num_contacts", "feature", "restitution_bias", "c0", "penalty", "lambda"):
        assert np.array_equal(getattr(before, "m_" + f)[:m], getattr(after, "m_" + f)[:m]), f
