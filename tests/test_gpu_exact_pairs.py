"""The exact collider's two forms: lists of up to 16,384 pairs take box pairs
on sixteen lanes each, longer lists a pair a thread.

The same pairs - boxes touching within rounding along a face or an edge axis,
clipped to polygons of three to eight vertices or to a support point,
separated by a hair, and sphere pairs - are decided once in a short list
(pair counts that fill a half, both and several warps) and once ahead of enough
touching boxes to make the list long. Every manifold must be bitwise the same,
and its topology the oracle's.
"""
import importlib
import math

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu

LONG = 16384  # narrowphase.cu kGroupMax


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def rotation(q):
    x, y, z, w = q
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])


def touching_pairs(scenes, count, filler, seed=11):
    """`count` pairs around x = 0, 12, 24, ..., then `filler` box pairs that
    touch within rounding (undecided in f32)."""
    s = scenes.Scene("touching")
    s.params = dict(gravity=0.0, iterations=1)
    rng = np.random.default_rng(seed)

    def quat(kind):
        if kind == 0:
            return np.array([0.0, 0.0, 0.0, 1.0])
        v = rng.normal(size=4)
        return (v / np.linalg.norm(v)).astype(np.float32).astype(np.float64)

    for k in range(count):
        at = np.array([12.0 * k, 0.0, 0.0])
        if k % 8 == 7:
            s.sphere(1.0, 100.0, 0.5, at)
            s.box((1.0, 1.4, 0.8), 100.0, 0.5, at + (0.9 + 1e-3 * (k % 3), 0.1, 0.0))
            continue
        ha, hb = rng.uniform(0.3, 1.0, 3), rng.uniform(0.3, 1.0, 3)
        qa, qb = quat(k % 4), quat(k % 3)
        if k % 2:  # B turned about the touching axis of A: faces of three to eight clipped vertices
            turn = (0.0, 1e-3, 0.5, math.pi / 4, 1.0)[k % 5]
            axis = np.eye(3)[k % 3] * math.sin(turn / 2)
            x, y, z, w = qa
            v, c = axis, math.cos(turn / 2)
            qb = np.concatenate([w * v + c * qa[:3] + np.cross(qa[:3], v), [w * c - qa[:3] @ v]])
            qb = (qb / np.linalg.norm(qb)).astype(np.float32).astype(np.float64)
        Ra, Rb = rotation(qa), rotation(qb)
        if k % 5 == 4:  # an edge axis
            n = np.cross(Ra[:, k % 3], Rb[:, (k + 1) % 3])
            n = n / np.linalg.norm(n) if np.linalg.norm(n) > 1e-2 else Ra[:, 2]
        else:
            n = Ra[:, k % 3] if k % 2 else Rb[:, k % 3]
        gap = (0.0, -1e-8, 1e-8, -3e-3)[k % 4]
        reach = np.abs(n @ Ra) @ ha + np.abs(n @ Rb) @ hb + gap
        side = np.cross(n, (0.3, 0.5, 0.8)) * rng.uniform(-0.4, 0.4)
        s.box(2 * ha, 100.0, 0.5, at, quat=tuple(qa))
        s.box(2 * hb, 100.0, 0.5, at + n * reach + side, quat=tuple(qb))
    for k in range(filler):
        at = (3.0 * (k % 200), 40.0 + 3.0 * (k // 200), 0.0)
        s.box((1.0, 1.0, 1.0), 100.0, 0.5, at)
        s.box((1.0, 1.0, 1.0), 100.0, 0.5, (at[0] + 1.0 - 1e-8, at[1], 0.0))
    return s


def random_pairs(scenes, abi, count, filler, seed=5):
    """Overlapping boxes at random poses; under the materials model's contact
    skin all of them go to the exact collider (faces clipped to nothing and
    support points among them)."""
    s = scenes.Scene("random")
    s.params = dict(gravity=0.0, iterations=1, contact_model=abi.CONTACT_MATERIALS)
    rng = np.random.default_rng(seed)
    for k in range(count):
        at = np.array([12.0 * (k % 64), 12.0 * (k // 64), -60.0])
        for side in range(2):
            v = rng.normal(size=4)
            q = (v / np.linalg.norm(v)).astype(np.float32).astype(np.float64)
            s.box(rng.uniform(0.1, 2.0, 3), 100.0, 0.5, at + side * rng.normal(0.0, 0.6, 3), quat=tuple(q))
    for k in range(filler):
        at = (3.0 * (k % 200), 40.0 + 3.0 * (k // 200), 0.0)
        s.box((1.0, 1.0, 1.0), 100.0, 0.5, at)
        s.box((1.0, 1.0, 1.0), 100.0, 0.5, (at[0] + 1.0 - 1e-8, at[1], 0.0))
    return s


def step(abi, backend_mod, s):
    gpu = backend_mod.GpuBackend(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY))
    gpu.pack(s.world())
    gpu.set_profiling(True)
    gpu.step(1)
    gpu.idle()
    exact = gpu.last_profile["np_exact"]
    out = gpu.read_state(manifolds=True)
    gpu.destroy()
    return out, exact


@pytest.mark.parametrize("kind,count", [("touching", 1), ("touching", 2), ("touching", 3), ("touching", 33),
                                        ("touching", 400), ("random", 4000)])
def test_short_and_long_lists_agree(abi, scenes, backend_mod, kind, count):
    make = (lambda f: touching_pairs(scenes, count, f)) if kind == "touching" else \
        (lambda f: random_pairs(scenes, abi, count, f))
    s = make(0)
    short, n_short = step(abi, backend_mod, s)
    long_, n_long = step(abi, backend_mod, make(LONG + 5))
    assert 0 < n_short <= LONG < n_long
    m = short.m_count
    assert m > 0 and m <= count and np.all(long_.m_body_a[:m] < 2 * count)
    for f in ("body_a", "body_b", "num_contacts", "basis", "friction", "feature", "r_a", "r_b", "c0"):
        assert np.array_equal(getattr(short, "m_" + f)[:m], getattr(long_, "m_" + f)[:m]), f
    ref = Oracle(abi.default_params(**s.params, body_order=abi.ORDER_PRIORITY), s.world())
    ref.step(1)
    assert short.manifold_dict() == ref.state().manifold_dict()
