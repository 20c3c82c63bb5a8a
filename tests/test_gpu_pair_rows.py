"""Rows of the broad phase longer than a warp's scratch row: a step re-enumerates
more than 128 partners of lower index, rank-sorted in shared memory up to 512 and
in place beyond; the allocation-free query does so beyond 64.

A bundle of thin rods whose bounding spheres all overlap, in no spatial order, so
that body k has k partners of lower index and none of the bodies is large; the
thicker rods touch their neighbours. A step's pairs and manifold topology are the
oracle's, on the second step with the first one's manifolds looked up among them.
"""
import importlib

import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


def bundle(scenes, rods, seed=2):
    s = scenes.Scene("bundle")
    rng = np.random.default_rng(seed)
    side = int(np.ceil(np.sqrt(rods)))
    for k in rng.permutation(side * side)[:rods]:
        t = 0.03 if rng.random() < 0.3 else 0.01
        s.box((1.0, t, t), 500.0, 0.5, (0.0, 0.024 * (k % side - side / 2), 0.024 * (k // side - side / 2)))
    return s


@pytest.mark.parametrize("longest", [127, 128, 129, 511, 512, 513, 700])
def test_rows_of_a_step(abi, scenes, backend_mod, longest):
    s = bundle(scenes, longest + 1)
    params = abi.default_params(gravity=0.0, iterations=1, body_order=abi.ORDER_PRIORITY)
    gpu = backend_mod.GpuBackend(params)
    gpu.pack(s.world())
    o = Oracle(params, s.world())
    for _ in range(2):
        gpu.step(1)
        o.step(1)
        gpu.idle()
        pairs, ref = np.asarray(gpu.read_pairs()), np.asarray(o.pairs())
        assert np.bincount(ref[0]).max() == longest
        assert np.array_equal(pairs, ref)
        out = gpu.read_state(manifolds=True)
        assert out.m_count > longest // 8 and out.manifold_dict() == o.state().manifold_dict()
    gpu.destroy()


@pytest.mark.parametrize("longest", [63, 64, 65, 128, 511, 512, 513, 700])
def test_rows_of_the_static_query(scenes, backend_mod, longest):
    torch = pytest.importorskip("torch")
    w = bundle(scenes, longest + 1).world()
    n = w.n_bodies
    want = np.concatenate([(a << 32) | np.arange(a, dtype=np.int64) for a in range(n)])
    dev = torch.device("cuda", torch.cuda.current_device())
    pos, radius = (torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (w.pos, w.radius))
    keys = torch.full((len(want) + 8,), -1, dtype=torch.int64, device=dev)
    count = torch.zeros(1, dtype=torch.int32, device=dev)
    cell = 2.0 * float(w.radius.max()) * (1 + 1e-6) + 1e-9
    backend_mod.overlap_pairs_static(n, pos.data_ptr(), radius.data_ptr(), 0, cell, keys.data_ptr(), keys.numel(),
                                     count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(count.item()) == len(want)
    assert np.array_equal(keys[:len(want)].cpu().numpy(), want) and int(keys[len(want)].item()) == -1
