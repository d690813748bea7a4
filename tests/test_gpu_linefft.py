"""The one-exchange line transforms against NumPy: every length with a plan as rows and as columns (paired with another,
column counts that are not a multiple of a tile among them), and Bluestein's on each work length at its smallest and
largest line, forward and inverse. Bounds: 1e-12 of the maximum in float64 and 2e-6 rel-L2 in float32, as the transforms'
other tests."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")

LENGTHS = [128, 160, 192, 200, 240, 250, 256, 300, 320, 360, 384, 400, 450, 480, 500, 512, 576, 600, 640, 720, 750, 768,
           800, 900, 960, 1024]
# prime factors above 64 (Bluestein), work lengths 256 to 1024: the smallest and largest lines of each, and odd counts
BLUESTEIN = [(67, 127), (71, 73), (134, 251), (131, 9), (257, 509), (262, 331), (511, 67)]


@pytest.mark.parametrize("nx,ny", list(zip(LENGTHS, LENGTHS[5:] + LENGTHS[:5])) + BLUESTEIN + [(45, 500), (512, 33)])
def test_against_numpy(nx, ny):
    engine = sk.Engine.require()
    rng = np.random.default_rng(nx * 1000 + ny)
    x = rng.normal(size=(3, nx, ny)) + 1j * rng.normal(size=(3, nx, ny))
    for inverse in (False, True):
        ref = np.fft.ifft2(x) if inverse else np.fft.fft2(x)
        y = engine.fft2(x, inverse, 64)
        assert np.abs(y - ref).max() <= 1e-12 * np.abs(ref).max()
        assert O.rel_l2(engine.fft2(x, inverse, 32), ref) <= 2e-6
