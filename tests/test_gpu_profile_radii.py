"""The full projection P_inf(rho) at radii from one ten-millionth of an angstrom down, where the integral form of K0 and K1
needs ever more points: the ratio of two elements' evaluations by a network whose embeddings are all alike, against the
oracle's Bessel functions, to 1e-12 as at ordinary radii. Radii past the Bessel functions' reach and infinite ones are
refused."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.fixture(scope="module")
def net():
    made = sk.Surrogate([6, 79], n_samples=1024, steps=1, batch=1024)
    p = np.random.default_rng(5).normal(0, 0.3, 11249).astype(np.float32)
    p[:103 * 16] = 0.0
    made.parameters(set_to=p, mean_std=(0.0, 1.0))
    return made


@pytest.mark.parametrize("rho", [1e-7, 1e-8, 1e-9, 1e-11, 1e-30, 1e-60, 1e-200])
def test_small(net, rho):
    r = np.array([rho])
    values = {z: net.evaluate(np.full(1, z), r, np.array([-1.0]), np.array([1.0]))[0] for z in (1, 6, 79, 103)}
    full = {z: float(O.infinite_profile(z, rho)) for z in values}
    assert abs(values[6]) > 0
    for z in (1, 79, 103):
        assert abs(values[z] / values[6] / (full[z] / full[6]) - 1) <= 1e-12


@pytest.mark.parametrize("rho", [1e7, 1e300, np.inf, np.nan])
def test_refused(net, rho):
    with pytest.raises(sk.SimulatoError):
        net.evaluate(np.array([6, 6]), np.array([1.0, rho]), np.array([-1.0, -1.0]), np.array([1.0, 1.0]))
    assert np.isfinite(net.evaluate(np.array([6]), np.array([4000.0]), np.array([-1.0]), np.array([1.0]))).all()
