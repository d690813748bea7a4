"""How exact the float32 transforms are, beside the bounds of the other tests, which leave room for a loss of several
times. A transform of N random values rounds at each of about log2 N levels: an error of at most 0.65 u sqrt(log2 N),
u = 2^-24, sqrt(2) times that in two dimensions (the constants' rounding included: twiddles twice as far off as rounding
to nearest puts them are outside). What every slice does alike shows in the energy: constants whose mean modulus is not
1, or 1/(nx ny) rounded to float32 (2.2e-8 off at 640^2), take the same share of it each time. A mean error of 6e-9 of the
energy a transform is 1e-6 after 40 slices of four transforms."""

import math

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")

LENGTHS = [128, 160, 192, 200, 240, 250, 256, 300, 320, 360, 384, 400, 450, 480, 500, 512, 576, 600, 640, 720, 750, 768,
           800, 900, 960, 1024]


@pytest.mark.parametrize("n", LENGTHS)
def test_transform(n):
    engine = sk.Engine.require()
    rng = np.random.default_rng(n)
    x = (rng.normal(size=(2, n, n)) + 1j * rng.normal(size=(2, n, n))).astype(np.complex64).astype(np.complex128)
    bound = 0.65 * 2.0 ** -24 * math.sqrt(2 * math.log2(n))
    for inverse in (False, True):
        ref = np.fft.ifft2(x) if inverse else np.fft.fft2(x)
        got = engine.fft2(x, inverse, 32)
        assert O.rel_l2(got, ref) <= bound
        if not inverse:  # (the inverse's 1 / n^2 is one float32 factor)
            assert abs(np.sum(np.abs(got) ** 2) / np.sum(np.abs(ref) ** 2) - 1) <= 4e-8


@pytest.mark.parametrize("n", [384, 500, 640])
def test_energy_of_jobs(n):
    slices = 40
    rng = np.random.default_rng(n)
    grid = O.Grid(n, n, 0.061 * n, 0.061 * n)
    values = rng.uniform(0, 30, (slices, n, n))
    wave = O.build_probe(O.ProbeSpec(200e3, 20.0), grid, (7.3, 5.1))
    ref = O.multislice(wave, [O.transmission(v, 200e3, grid) for v in values], [2.0] * slices, 200e3, grid)[-1]
    pot = sk.ProjectedPotential(sk.Grid(n, n, 0.061 * n, 0.061 * n), values, [2.0] * slices)
    table = sk.JobTable()
    table.add_probe(pot, sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0)), (7.3, 5.1))
    got = table.run()[0][0]
    assert abs(got.sum() / np.sum(np.abs(ref) ** 2) - 1) <= 1e-6


@pytest.mark.parametrize("n", [200, 256, 500, 640])
def test_energy_of_plane_waves(n):
    """A plane wave's energy is in one value of its transform. Rounded to float32 once a slice, that would leave an error
    of about 2^-24 sqrt(slices / 3) in the energy; it is less, as the transforms' levels don't round it one by one."""
    slices, draws = 40, 6
    grid = O.Grid(n, n, 0.061 * n, 0.061 * n)
    errors = []
    for draw in range(draws):
        values = np.random.default_rng(1000 * n + draw).uniform(0, 30, (slices, n, n))
        wave = np.ones((n, n), complex)
        ref = O.multislice(wave, [O.transmission(v, 200e3, grid) for v in values], [2.0] * slices, 200e3, grid)[-1]
        pot = sk.ProjectedPotential(sk.Grid(n, n, 0.061 * n, 0.061 * n), values, [2.0] * slices)
        table = sk.JobTable()
        table.add_plane_wave(pot, 200e3)
        got = table.run()[0][0]
        errors.append((got.sum() / got.size) / np.mean(np.abs(ref) ** 2) - 1)
    assert np.sqrt(np.mean(np.square(errors))) <= 2.0 ** -24 * math.sqrt(slices / 3)
