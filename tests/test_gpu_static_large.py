"""The allocation-free overlap query with bodies wider than its cell: each is
tested against every body before it, 1,024 at a time, by a block that takes the
next one from a list in no order. Keys and count are those of a direct f64 test
of all pairs, and a query of which one body in twenty is that wide costs less
than nine times one without such bodies (6 measured; 13 with a quarter of the
threads)."""
import importlib
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend_mod():
    return importlib.import_module("avbd-sandbox_gb300.backend")


@pytest.fixture(scope="module")
def torch():
    return pytest.importorskip("torch")


def cloud(n, large, seed, side):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-side / 2, side / 2, (n, 3))
    radius = rng.uniform(0.3, 0.8, n)
    radius[[i for i in large if i < n]] = 3.0
    return pos, radius, (rng.random(n) < 0.7).astype(np.int32)


def expected(pos, radius, dynamic):
    """Keys (a << 32 | b, b < a) of the overlapping pairs, ascending."""
    keys = []
    for a in range(len(pos)):
        d, r = pos[a] - pos[:a], radius[a] + radius[:a]
        hit = ((d * d).sum(axis=1) <= r * r) & ((dynamic[a] != 0) | (dynamic[:a] != 0))
        keys.append((a << 32) | np.nonzero(hit)[0].astype(np.int64))
    return np.concatenate(keys)


class Query:
    def __init__(self, torch, backend_mod, pos, radius, dynamic, capacity):
        self.torch, self.be, self.n = torch, backend_mod, len(pos)
        dev = torch.device("cuda", torch.cuda.current_device())
        self.args = [torch.from_numpy(np.ascontiguousarray(x)).to(dev) for x in (pos, radius, dynamic)]
        self.keys = torch.full((capacity,), -1, dtype=torch.int64, device=dev)
        self.count = torch.zeros(1, dtype=torch.int32, device=dev)

    def __call__(self, calls=1):
        p, r, d = (x.data_ptr() for x in self.args)
        t = time.perf_counter()
        for _ in range(calls):
            self.be.overlap_pairs_static(self.n, p, r, d, 1.61, self.keys.data_ptr(), self.keys.numel(),
                                         self.count.data_ptr(), self.torch.cuda.current_stream().cuda_stream)
        self.torch.cuda.synchronize()
        return time.perf_counter() - t


@pytest.mark.parametrize("n", [1, 2, 1024, 1025, 1026, 2049, 5000])
@pytest.mark.parametrize("large", [(0, 1), (1023, 1024, 1025, 2048), tuple(range(0, 5000, 3))])
def test_pairs_of_large_bodies(torch, backend_mod, n, large):
    pos, radius, dynamic = cloud(n, large, n + len(large), 1.2 * n ** (1 / 3) + 1.0)
    want = expected(pos, radius, dynamic)
    q = Query(torch, backend_mod, pos, radius, dynamic, len(want) + 16)
    q()
    assert int(q.count.item()) == len(want)
    assert np.array_equal(q.keys[:len(want)].cpu().numpy(), want)


def test_large_bodies_cost(torch, backend_mod):
    q = [Query(torch, backend_mod, *cloud(20000, large, 9, 30.0), 600 * 20000)
         for large in ((), np.random.default_rng(1).permutation(20000)[:1000])]
    few, many = (sorted(x(20) for _ in range(5))[2] for x in q)
    assert many < 9.0 * few, many / few
