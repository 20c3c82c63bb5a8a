"""Scenes whose stiffest joint or spring cannot make an FP64 body run solve
kernels without an FP64 path (avbd_pack's bound). A body on one joint or spring
whose stiffness lies just below and just above the ratio, with the penalty
there at once or reached in the middle of a run, is an FP64 body exactly when
its penalty exceeds fp64_ratio_threshold * m / dt^2.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def hanging(scenes, kind, stiffness, rest=2.0):
    """The body, 2 kg, on a joint to the world, a joint to a static box or a spring."""
    s = scenes.Scene("hanging")
    s.box((1.0, 1.0, 1.0), 0.0, 0.5, (0.0, 0.0, 3.0))
    s.box((0.1, 0.1, 0.1), 2000.0, 0.5, (0.0, 0.0, 0.0))
    if kind == "world":
        s.joint(-1, 1, (0.0, 0.0, 0.5), (0.0, 0.0, 0.5), stiffness_lin=stiffness)
    elif kind == "joint":
        s.joint(0, 1, (0.0, 0.0, -2.5), (0.0, 0.0, 0.5), stiffness_lin=stiffness)
    elif kind == "spring":
        s.spring(1, 0, (0.0, 0.0, 0.05), (0.0, 0.0, -0.5), stiffness, rest=rest)
    return s


@pytest.mark.parametrize("kind", ["world", "joint", "spring", "hard"])
@pytest.mark.parametrize("ratio", [1e3, 1e5])
@pytest.mark.parametrize("above", [False, True])
def test_stiffness_around_the_ratio(abi, scenes, backend_mod, kind, ratio, above):
    kw = dict(gravity=-9.81, iterations=5, body_order=abi.ORDER_PRIORITY, fp64_ratio_threshold=ratio)
    line = ratio * 2.0 * 60.0 ** 2
    k = line * (1.0 + (1e-3 if above else -1e-3))
    if kind == "hard":  # a hard joint counts with the largest penalty
        kw["penalty_max"] = k
        s = hanging(scenes, "joint", float("inf"))
    else:
        s = hanging(scenes, kind, k)
    w = s.world()
    if w.n_joints:
        w.j_penalty_lin[:] = 10.0 * k  # (capped at the stiffness)
    gpu = backend_mod.GpuBackend(abi.default_params(**kw))
    gpu.pack(w)
    gpu.set_profiling(True)
    for step in range(3):
        gpu.step(1)
        # a soft joint's penalty starts the step at gamma (0.999) times the last one's end, a hard one counts at its cap
        assert gpu.last_profile["fp64_bodies"] == (1 if above and (step == 0 or kind in ("spring", "hard")) else 0)
    gpu.idle()
    assert np.all(np.isfinite(gpu.read_state().pos))
    gpu.destroy()


@pytest.mark.parametrize("kind", ["joint", "spring"])
def test_a_penalty_that_passes_the_ratio_later(abi, scenes, backend_mod, kind):
    line = 1e3 * 2.0 * 60.0 ** 2
    params = abi.default_params(gravity=-200.0, iterations=5, body_order=abi.ORDER_PRIORITY, fp64_ratio_threshold=1e3,
                                spring_stiffness_ramp=1, beta_lin=1.2e8)
    gpu = backend_mod.GpuBackend(params)
    gpu.pack(hanging(scenes, kind, 3.0 * line, rest=2.45).world())
    gpu.set_profiling(True)
    start, seen = 0.0, []  # of the next step: the penalty its warm start begins from
    for _ in range(40):
        gpu.step(1)
        seen.append(gpu.last_profile["fp64_bodies"])
        assert seen[-1] == (1 if 0.999 * start > line else 0)
        out = gpu.read_state()
        start = float(out.j_penalty_lin.max()) if kind == "joint" else float(out.s_penalty[0])
    gpu.destroy()
    assert seen[0] == 0 and seen[1] == 0 and seen[-1] == 1
