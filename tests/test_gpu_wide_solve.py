"""The colour-phase solve's two FP32 forms give the same bits.

A colour of C lane chunks (128 lanes each) is solved in the wide form, four
threads a lane, when 4 C fits the grid, else in the staged form. With one solve
block per SM instead of three the line lies at a third of the chunks, so
colours between the two lines change form between the two runs; the body
state and every multiplier and penalty must not.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "quat", "vel", "omega", "m_penalty", "m_lambda", "m_stick", "j_penalty_lin", "j_lambda_lin",
          "j_penalty_ang", "j_lambda_ang", "j_broken")


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


@pytest.mark.parametrize("scene,materials,steps", [("pyramid", False, 14), ("pyramid", True, 14), ("wall", False, 4)])
def test_forms_agree(abi, scenes, backend_mod, scene, materials, steps):
    if scene == "pyramid":  # 7,714 cubes in about five colours of 48 chunks and more
        s = scenes.pyramid(layers=28)
    else:  # 10,000 bricks and 19,800 bonds
        s = scenes.brick_wall(cols=100, rows=100)
        s.b["pos"][-1] = (0.0, -0.6, 12.0)
    w = s.world()
    kw = dict(s.params, body_order=abi.ORDER_PRIORITY)
    if materials:
        kw["contact_model"] = abi.CONTACT_MATERIALS
        w.set_materials(static_friction=0.7, dynamic_friction=0.5, restitution=0.1)
    outs = []
    for blocks in (1, 3):
        gpu = backend_mod.GpuBackend(abi.default_params(**kw, blocks_per_sm=blocks))
        gpu.pack(w)
        gpu.set_profiling(True)
        gpu.step(steps)
        gpu.idle()
        p = gpu.last_profile
        chunks = p["lanes_per_body"] * w.n_bodies / 128 / p["colors"]
        assert 152 < 4 * chunks < 3 * 152 * 2, chunks  # the mean colour lies between the lines, or near the upper one
        outs.append(gpu.read_state(manifolds=True))
        gpu.destroy()
    assert scene == "wall" or outs[0].m_count > w.n_bodies // 4
    assert outs[0].m_count == outs[1].m_count
    for f in FIELDS:
        assert np.array_equal(getattr(outs[0], f), getattr(outs[1], f)), f
