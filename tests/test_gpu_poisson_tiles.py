"""Poisson noise drawn in the order of the means within tiles of 2048 values, against the oracle's per-value streams, bit
for bit: counts around a tile, means of every bin (0, below 1, each whole part up to 10, above), several samples, and in
place."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("count", [1, 255, 2047, 2048, 2049, 6000])
def test_equals_the_streams(count):
    rng = np.random.default_rng(count)
    values = rng.uniform(-0.05, 1.0, count) ** 3 * 14.0
    values[rng.integers(0, count, max(1, count // 10))] = 0.0
    m = sk.ScanMeasurement([1, count], [], values)
    ref = O.poisson_noise_streams(values, 1.5, 77, samples=2)
    got = m.poissonNoise(1.5, samples=2, seed=77)
    for s in range(2):
        assert np.array_equal(np.asarray(got[s].values), np.asarray(ref[s]).ravel())
