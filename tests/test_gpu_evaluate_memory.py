"""Evaluating many queries once does not keep their device memory (44 bytes each) for the life of the engine; the values are
those of the same queries in parts, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")
torch = pytest.importorskip("torch")


def test_memory_comes_back():
    n = 7_000_000
    engine = sk.Engine(0)
    net = sk.Surrogate([6, 79], n_samples=1024, steps=1, batch=1024, engine=engine)
    rng = np.random.default_rng(3)
    z, rho = rng.choice([6, 79], n).astype(np.int32), rng.uniform(0.05, 5.0, n)
    zl = rng.uniform(-3, 0, n)
    zu = zl + 1.0
    some = net.evaluate(z[:1000], rho[:1000], zl[:1000], zu[:1000])
    before = torch.cuda.mem_get_info(0)[0]
    got = net.evaluate(z, rho, zl, zu)
    assert before - torch.cuda.mem_get_info(0)[0] <= 100 << 20
    assert np.array_equal(got[:1000], some)
    assert np.array_equal(net.evaluate(z[-1000:], rho[-1000:], zl[-1000:], zu[-1000:]), got[-1000:])
