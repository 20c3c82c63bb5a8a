"""Resting boxes: lists of pairs that nearly all touch take a pair a thread from
6,145 pairs on (narrowphase.cu kGroupMaxAlike), where sixteen lanes a pair cost
more, on the first step after a pack as later, with and without a contact skin
and under both contact models.

A list of 13,000 such pairs takes no longer than one of 17,000, which is past
the line of any list, and a box's contacts and motion are the same bits in
lists on both sides of the line.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OFFSETS = [0.02, 0.0, None]  # contact offset under the materials model; None: the plain model


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def resting(scenes, boxes):
    s = scenes.Scene("resting")
    scenes.add_ground(s, 0.5)
    rng = np.random.default_rng(3)
    size = rng.uniform(0.6, 1.2, (boxes, 3))
    for k in range(boxes):
        s.box(size[k], 500.0, 0.5, (2.2 * (k % 130 - 65), 2.2 * (k // 130 - 65), 0.5 * size[k, 2] - 0.009))
    return s


def run(abi, scenes, backend_mod, boxes, steps, offset):
    """The narrow phase's time of each step, and the state after them."""
    s = resting(scenes, boxes)
    w = s.world()
    if offset is not None:
        w.set_materials(static_friction=0.7, dynamic_friction=0.5, restitution=0.2, contact_offset=offset)
    gpu = backend_mod.GpuBackend(abi.default_params(
        gravity=-9.81, iterations=4, body_order=abi.ORDER_PRIORITY,
        contact_model=abi.CONTACT_CPU if offset is None else abi.CONTACT_MATERIALS))
    gpu.pack(w)
    gpu.set_profiling(True)
    ms = []
    for _ in range(steps):
        gpu.step(1)
        ms.append(gpu.last_profile["narrowphase_ms"])
    gpu.idle()
    exact = gpu.last_profile["np_exact"]
    out = gpu.read_state(manifolds=True)
    gpu.destroy()
    return ms, exact, out


@pytest.mark.parametrize("offset", OFFSETS)
def test_a_shorter_list_takes_no_longer(abi, scenes, backend_mod, offset):
    run(abi, scenes, backend_mod, 200, 2, offset)  # (the library is loaded and the clocks are up)
    short, n_short, _ = run(abi, scenes, backend_mod, 13000, 9, offset)
    long_, n_long, _ = run(abi, scenes, backend_mod, 17000, 9, offset)
    assert 6144 < n_short <= 16384 < n_long
    assert np.median(short) < 1.25 * np.median(long_)
    assert short[0] < 1.25 * long_[0]  # without a previous step's manifolds


@pytest.mark.parametrize("offset", OFFSETS)
@pytest.mark.parametrize("boxes", [6144, 6145, 8193])
def test_contacts_do_not_depend_on_the_line(abi, scenes, backend_mod, boxes, offset):
    _, exact, few = run(abi, scenes, backend_mod, 300, 3, offset)
    _, exact_many, many = run(abi, scenes, backend_mod, boxes, 3, offset)
    m = few.m_count
    assert exact == m == 300 and exact_many == many.m_count == boxes
    for f in ("body_a", "body_b", "num_contacts", "basis", "feature", "r_a", "r_b", "c0", "penalty", "lambda", "stick",
              "restitution_bias"):
        assert np.array_equal(getattr(few, "m_" + f)[:m], getattr(many, "m_" + f)[:m]), f
    for f in ("pos", "quat", "vel", "omega"):
        assert np.array_equal(getattr(few, f), getattr(many, f)[:301]), f
