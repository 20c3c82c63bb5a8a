"""State exchange on both sides of its size limit (2,048 bodies, joints or
springs): below it one kernel reads or writes the pinned copy of the whole
state, above it arrays are copied one by one. What was written comes back as
the device holds it (positions in f64, the rest of a body in f32), joints and
springs included, and a position that is not finite changes nothing at all.
"""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F64 = ("pos", "j_lambda_lin", "j_lambda_ang", "s_peak_strain")
F32 = ("quat", "vel", "omega", "prev_vel", "j_penalty_lin", "j_penalty_ang", "s_penalty")


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def world_of(scenes, bodies, joints, springs):
    """Boxes far apart in a row; joints and springs between neighbours."""
    sc = scenes.Scene("exchange")
    for i in range(bodies):
        sc.box((0.5, 0.5, 0.5), 500.0, 0.5, (2.0 * i, 0.0, 5.0))
    for j in range(joints):
        sc.joint(j % (bodies - 1), j % (bodies - 1) + 1, (1.0, 0.0, 0.0), (-1.0, 0.0, 0.0))
    for k in range(springs):
        sc.spring(k % (bodies - 1), k % (bodies - 1) + 1, (0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 100.0)
    return sc


@pytest.mark.parametrize("bodies,joints,springs", [(1, 0, 0), (33, 5, 3), (2048, 2048, 2048), (2049, 7, 3), (40, 2049, 3),
                                                   (40, 3, 2049)])
def test_round_trip(abi, scenes, backend_mod, bodies, joints, springs):
    gpu = backend_mod.GpuBackend(abi.default_params())
    w = world_of(scenes, bodies, joints, springs).world()
    gpu.pack(w)
    rng = np.random.default_rng(bodies + joints)
    host = gpu.read_state()
    for f in F64 + F32:
        a = getattr(host, f)
        if a is not None and a.size:
            setattr(host, f, a + rng.uniform(0.0, 1.0, a.shape))
    if joints:
        host.j_broken[::2] = 1
    if springs:
        host.s_broken[1::2] = 1
    gpu.write_state(host)
    back = gpu.read_state()
    bad = host.copy()
    bad.pos[bodies // 2, 2] = np.inf
    bad.vel[:] = 7.0
    if joints:
        bad.j_lambda_lin[:] = 7.0
    with pytest.raises(backend_mod.AvbdError) as e:
        gpu.write_state(bad)
    assert e.value.code == abi.AVBD_ERR_NAN and f"body {bodies // 2}:" in str(e.value)
    after = gpu.read_state()
    gpu.destroy()
    for got in (back, after):
        for f in F64:
            assert np.array_equal(getattr(got, f), getattr(host, f)), f
        for f in F32:
            assert np.array_equal(getattr(got, f), getattr(host, f).astype(np.float32).astype(np.float64)), f
        assert np.array_equal(got.j_broken, host.j_broken) and np.array_equal(got.s_broken, host.s_broken)


def test_no_positions_is_refused(abi, scenes, backend_mod):
    gpu = backend_mod.GpuBackend(abi.default_params())
    w = world_of(scenes, 5, 2, 1).world()
    gpu.pack(w)
    before = gpu.read_state()
    w.vel[:] = 3.0
    wc = w.c(with_manifolds=False)
    wc.bodies.pos = None
    assert gpu.L.avbd_write_state(gpu.h, ctypes.byref(wc)) == abi.AVBD_ERR_CUDA
    assert np.array_equal(gpu.read_state().vel, before.vel)
    gpu.destroy()
