"""The wide form of the colour-phase solve against the staged form where it meets
more than boxes in FP32: joints and springs under both contact models, FP64
bodies beside FP32 ones in a unit, a grabbed body, a group of more than a warp
among small ones, and a colour that is known to change form.

A fixed lane count turns the wide form off. With at most 16 constraints a body
both have groups of four lanes, so the states must agree bit for bit.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("pos", "quat", "vel", "omega")
FORCES = ("j_penalty_lin", "j_penalty_ang", "j_lambda_lin", "j_lambda_ang", "j_broken", "s_penalty", "s_peak_strain",
          "s_broken", "m_penalty", "m_lambda", "m_stick")


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def bridge(scenes, boxes):
    """Boxes on the ground in a row, light and heavy ones in turn, each jointed
    or sprung to the next: 4 contacts and up to 4 joints and springs a box."""
    s = scenes.Scene("bridge")
    scenes.add_ground(s, 0.5)
    first = [s.box((0.5, 0.5, 0.5), 60.0 if k % 2 else 600.0, 0.5, (0.6 * k, 0.02 * (k % 3), 0.25 - 1e-3))
             for k in range(boxes)]
    for k in range(boxes - 1):
        if k % 3 == 2:
            s.spring(first[k], first[k + 1], (0.3, 0.0, 0.0), (-0.3, 0.0, 0.0), 2000.0, rest=0.1)
        else:
            s.joint(first[k], first[k + 1], (0.3, 0.0, 0.0), (-0.3, 0.0, 0.0),
                    stiffness_ang=float("inf") if k % 3 else 0.0, fracture=50.0)
    return s


@pytest.mark.parametrize("materials", [False, True])
@pytest.mark.parametrize("grab", [None, 1, 6])
@pytest.mark.parametrize("ratio", [0.0, 1e5])
def test_forces_in_both_forms(abi, scenes, backend_mod, materials, grab, ratio):
    s = bridge(scenes, 90)
    w = s.world()
    kw = dict(gravity=-9.81, iterations=8, body_order=abi.ORDER_PRIORITY, fp64_ratio_threshold=ratio)
    if materials:
        kw["contact_model"] = abi.CONTACT_MATERIALS
        w.set_materials(static_friction=0.7, dynamic_friction=0.5, restitution=0.1)
    outs, fp64 = [], set()
    for lanes in (0, 4):
        gpu = backend_mod.GpuBackend(abi.default_params(**kw, lanes_per_body=lanes))
        gpu.pack(w)
        if grab is not None:
            gpu.set_grab(grab, (0.1, 0.0, 0.2), (3.0, 1.0, 1.5), 4000.0)
        gpu.set_profiling(True)
        for _ in range(6):
            gpu.step(1)
            p = gpu.last_profile
            fp64.add(p["fp64_bodies"])
            assert p["lanes_per_body"] == 4
        gpu.idle()
        outs.append(gpu.read_state(manifolds=True))
        gpu.destroy()
    assert fp64 == {0} if ratio == 0.0 else 0 < max(fp64) < 90  # (FP64 bodies beside FP32 ones)
    assert outs[0].m_count == outs[1].m_count > 0
    m = outs[0].m_count
    for f in STATE + FORCES:
        a, b = (getattr(o, f)[:m] if f.startswith("m_") else getattr(o, f) for o in outs)
        assert np.array_equal(a, b), f


@pytest.mark.parametrize("loads,bodies", [(6, 200), (9, 40)])
def test_a_wide_group_among_small_ones(abi, scenes, backend_mod, loads, bodies):
    """A plate with a group of 64 or 128 lanes shares its colour's first chunk
    with small bodies that touch nothing of it; they move as they do alone."""
    def small(s):
        return [s.box((0.5, 0.5, 0.5), 500.0, 0.5, (60.0 + 0.9 * (k // 2 % 20), 0.9 * (k // 40),
                                                    0.25 + 0.5 * (k % 2) - 1e-3))
                for k in range(bodies)]  # (two on each other: two colours)

    params = abi.default_params(gravity=-9.81, iterations=6, body_order=abi.ORDER_PRIORITY)
    outs = []
    for plate in (False, True):
        s = scenes.Scene("loads")
        scenes.add_ground(s, 0.6)
        free = small(s)
        if plate:
            side = 2.0 * loads + 2.0
            s.box((side, side, 0.5), 1000.0, 0.6, (0.0, 0.0, 0.25 - 1e-3))
            for k in range(loads * loads):
                s.box((1.0, 1.0, 1.0), 1000.0, 0.6, ((k % loads - (loads - 1) / 2) * 2.0,
                                                     (k // loads - (loads - 1) / 2) * 2.0, 1.0 - 2e-3))
        gpu = backend_mod.GpuBackend(params)
        gpu.pack(s.world())
        gpu.step(3)
        gpu.idle()
        out = gpu.read_state()
        colors, _ = gpu.read_coloring()
        gpu.destroy()
        outs.append([getattr(out, f)[free] for f in STATE])
        if plate:
            assert np.any(colors[free] == colors[bodies + 1])
    for f, a, b in zip(STATE, *outs):
        assert np.array_equal(a, b), f


def test_a_colour_that_changes_form(abi, scenes, backend_mod):
    """With one solve block an SM and with three, some colour of this scene is
    staged in the first run and wide in the second."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    s = scenes.pyramid(layers=28)
    outs = []
    for blocks in (1, 3):
        gpu = backend_mod.GpuBackend(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY,
                                                        blocks_per_sm=blocks))
        gpu.pack(s.world())
        gpu.step(14)
        gpu.idle()
        outs.append((gpu.read_state(manifolds=True), gpu.read_coloring()))
        gpu.destroy()
    (a, (colors, count)), (b, (other, _)) = outs
    assert np.array_equal(colors, other)
    m = a.m_count
    sides = np.zeros(a.n_bodies, np.int64)
    for side in (a.m_body_a[:m], a.m_body_b[:m]):
        np.add.at(sides, side, a.m_num_contacts[:m])
    lanes = 4 << np.maximum(0, np.ceil(np.log2(np.maximum(sides, 1) / 16.0))).astype(int)
    chunks = [-(-int(lanes[colors == c].sum()) // 128) for c in range(count)]
    assert any(sms < 4 * c <= 3 * sms for c in chunks), chunks
    for f in STATE + ("m_penalty", "m_lambda", "m_stick"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f
