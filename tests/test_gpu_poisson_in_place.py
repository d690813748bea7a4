"""Poisson noise written over its means (one sample, the device form), bit for bit the noise written beside them: counts
around a tile of 2048 values, and more tiles than blocks, so that a block goes on to further ones; both streams."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("count,stream", [(1, 0), (2047, 0), (2048, 0), (2049, 0), (16 * 148 * 2048 * 2 + 77, 0), (500, 1)])
def test_over_the_means(count, stream):
    from simulatokit_b200 import _lib as L
    engine = sk.Engine(0)
    L.check(engine.lib.simk_context_set_option(engine.handle, L.OPT_POISSON_STREAM, stream))
    rng = np.random.default_rng(count)
    means = torch.from_numpy(rng.uniform(-0.05, 1.0, count) ** 3 * 14.0).cuda()
    beside = torch.empty_like(means)
    at = [L.C.cast(L.C.c_void_p(t.data_ptr()), L.PD) for t in (means, beside)]
    torch.cuda.synchronize()
    for out in (at[1], at[0]):
        L.check(engine.lib.simk_poisson_noise_device(engine.handle, count, at[0], 1.5, 1, 77, out))
    engine.synchronize()
    assert torch.equal(means, beside) and float(beside.sum()) > 0
