"""The narrow phase's lists are worked on side by side, in units of a warp
that are dealt when they are fewer than the warps and claimed one by one when
there are more; a pair's contacts must not depend on it.

One cluster of overlapping boxes and spheres is stepped alone and as a batch
of copies. Every copy's contact geometry is bitwise the single cluster's, and
its topology the oracle's.
"""
import importlib

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def cluster(scenes, abi, bodies, materials, seed=17):
    s = scenes.Scene("cluster")
    s.params = dict(gravity=0.0, iterations=1)
    if materials:
        s.params["contact_model"] = abi.CONTACT_MATERIALS
    rng = np.random.default_rng(seed)
    side = max(2.0, 0.7 * bodies ** (1 / 3))
    for k in range(bodies):
        at = rng.uniform(-side, side, 3)
        q = rng.normal(size=4) if k % 3 else np.array([0.0, 0.0, 0.0, 1.0])  # aligned ones: tied face axes
        q = (q / np.linalg.norm(q)).astype(np.float32).astype(np.float64)
        if k % 9 == 8:
            s.sphere(float(rng.uniform(0.6, 1.4)), 100.0, 0.5, at)
        else:
            s.box(rng.uniform(0.5, 1.5, 3) if k % 2 else (1.0, 1.0, 1.0), 100.0, 0.5, at, quat=tuple(q))
    return s


def step(abi, backend_mod, params, world):
    gpu = backend_mod.GpuBackend(abi.default_params(**params, body_order=abi.ORDER_PRIORITY))
    gpu.pack(world)
    gpu.set_profiling(True)
    gpu.step(1)
    gpu.idle()
    p = gpu.last_profile
    out = gpu.read_state(manifolds=True)
    gpu.destroy()
    return out, (p["np_exact"] + 1) // 2 + (p["np_face"] + 31) // 32 + (p["np_edge"] + 31) // 32


@pytest.mark.parametrize("bodies,copies,materials", [(40, 1, False), (60, 40, False), (60, 900, False), (40, 1, True),
                                                     (60, 120, True)])
def test_contacts_do_not_depend_on_the_lists(abi, scenes, backend_mod, bodies, copies, materials):
    s = cluster(scenes, abi, bodies, materials)
    one, units = step(abi, backend_mod, s.params, s.world())
    assert 0 < units < 152 * 8
    ref = Oracle(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY), s.world())
    ref.step(1)
    assert one.m_count > bodies // 2 and one.manifold_dict() == ref.state().manifold_dict()
    if copies == 1:
        return
    many, units = step(abi, backend_mod, s.params, scenes.batch_worlds([s.world() for _ in range(copies)]))
    assert copies < 100 or units > 152 * 8
    m = one.m_count
    assert many.m_count == copies * m
    off = np.repeat(np.arange(copies) * bodies, m)
    assert np.array_equal(many.m_body_a[:copies * m], np.tile(one.m_body_a[:m], copies) + off)
    assert np.array_equal(many.m_body_b[:copies * m], np.tile(one.m_body_b[:m], copies) + off)
    for f in ("num_contacts", "basis", "friction", "feature", "r_a", "r_b", "c0", "restitution_bias"):
        a, b = getattr(one, "m_" + f)[:m], getattr(many, "m_" + f)[:copies * m].reshape((copies, m) + getattr(one, "m_" + f).shape[1:])
        assert np.all(b == a[None]), f


@pytest.mark.parametrize("bodies", [12, 40, 120])
def test_materials_merge_on_lanes_and_by_threads(abi, scenes, backend_mod, bodies):
    """Under the materials model a box pair's contacts claim the previous
    step's on sixteen lanes, in lists of more than 16,384 pairs by a thread:
    the same claims, so the same bits over several steps."""
    outs = []
    for filler in (0, 16400):
        s = cluster(scenes, abi, bodies, True, seed=3)
        s.params.update(gravity=-9.81, iterations=4)
        for k in range(filler):
            at = np.array([40.0 + 4.0 * (k % 128), 4.0 * (k // 128), 0.0])
            s.box((1.0, 1.0, 1.0), 100.0, 0.5, at)
            s.box((1.0, 1.0, 1.0), 100.0, 0.5, at + (0.0, 0.0, 0.99))
        w = s.world()
        w.set_materials(static_friction=0.7, dynamic_friction=0.5, restitution=0.2, contact_offset=0.02)
        gpu = backend_mod.GpuBackend(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY))
        gpu.pack(w)
        gpu.set_profiling(True)
        gpu.step(6)
        gpu.idle()
        assert (gpu.last_profile["np_exact"] > 16384) == (filler > 0)
        outs.append(gpu.read_state(manifolds=True))
        gpu.destroy()
    short, long_ = outs
    m = short.m_count
    assert m > 0 and np.all(long_.m_body_a[:m] < bodies)
    for f in ("body_a", "body_b", "num_contacts", "basis", "feature", "r_a", "r_b", "c0", "penalty", "lambda", "stick",
              "restitution_bias"):
        assert np.array_equal(getattr(short, "m_" + f)[:m], getattr(long_, "m_" + f)[:m]), f
    assert np.array_equal(short.pos, long_.pos[:bodies]) and np.array_equal(short.quat, long_.quat[:bodies])
