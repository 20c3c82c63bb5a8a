"""The materials merge on sixteen lanes with an old contact that is not a
number: a new contact claims the nearest old one in the serial merge's sense,
in which nothing is less than NaN - a NaN distance is kept when it is the first
candidate, and passed over after a finite one.

Two boxes face to face, no feature of the old manifold known to the new one, so
that every claim goes by distance; the old penalties tell the claims apart.
"""
import importlib

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("lost", [(0,), (1,), (3,), (1, 2), (0, 3), (0, 1, 2, 3)])
def test_claims_around_a_nan(abi, scenes, backend_mod, lost, reverse):
    s = scenes.Scene("pair")
    s.box((2.0, 2.0, 1.0), 0.0, 0.5, (0.0, 0.0, 0.0))
    s.box((1.0, 1.0, 1.0), 500.0, 0.5, (0.1, 0.05, 0.999))
    params = abi.default_params(gravity=0.0, iterations=0, body_order=abi.ORDER_PRIORITY,
                                contact_model=abi.CONTACT_MATERIALS)
    o = Oracle(params, s.world())
    o.step(1)
    state = o.state().round_to_device()
    assert state.m_count == 1 and state.m_num_contacts[0] == 4
    state.m_feature[0, :4] += 100
    state.m_stick[0, :4] = 0
    state.m_penalty[0, :4] = np.array([1e3, 2e3, 3e3, 4e3])[:, None]
    if reverse:
        for a in (state.m_r_a, state.m_r_b):
            a[0, :4] = a[0, 3::-1].copy()
    state.m_r_a[0, list(lost)] = np.nan
    ref = Oracle(params, state)
    ref.step(1)
    want = ref.state()
    gpu = backend_mod.GpuBackend(params)
    gpu.pack(state)
    gpu.step(1)
    gpu.idle()
    got = gpu.read_state(manifolds=True)
    gpu.destroy()
    assert got.manifold_dict() == want.manifold_dict()
    # one f32 rounding of gamma times the claimed penalty (1 when nothing was claimed)
    assert np.allclose(got.m_penalty[0, :4], want.m_penalty[0, :4], rtol=2.0 ** -23, atol=0.0)
