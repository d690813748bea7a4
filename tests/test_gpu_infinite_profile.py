"""The full projection P_inf(rho) on the device against the oracle's Bessel functions. The surrogate's evaluation is
P_inf(rho) F with F from the network; with every embedding alike F does not depend on the element, so the ratio of two
elements' evaluations at one (rho, zl, zu) is the ratio of their full projections. Each is good to about 1e-13 (the
rounding of x cosh u in the exponentials, x up to 100 where a term still counts): 1e-12 for the ratio."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("n", [1, 127, 1000])
def test_ratio_of_full_projections(n):
    net = sk.Surrogate([6, 79], n_samples=1024, steps=1, batch=1024)
    rng = np.random.default_rng(5)
    p = rng.normal(0, 0.3, 11249).astype(np.float32)
    p[:103 * 16] = 0.0
    net.parameters(set_to=p, mean_std=(0.0, 1.0))
    rho = np.exp(rng.uniform(np.log(0.005), np.log(8.0), n))
    zl = rng.uniform(-3, 0, n)
    zu = zl + rng.uniform(0.5, 4, n)
    values = {z: net.evaluate(np.full(n, z), rho, zl, zu) for z in (1, 6, 38, 79, 103)}
    full = {z: np.array([O.infinite_profile(z, r) for r in rho]) for z in values}
    used = np.abs(values[6]) > 0
    assert used.mean() > 0.9
    for z in (1, 38, 79, 103):
        a, b = values[z][used] / values[6][used], full[z][used] / full[6][used]
        assert np.max(np.abs(a / b - 1)) <= 1e-12
