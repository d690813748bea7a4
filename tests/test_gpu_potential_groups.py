"""The builder's groups of slices: empty slices between occupied ones, many elements in one slice, and a slice whose delta
images exceed one batch (20 elements at 1024^2: 16 images a batch), against the oracle's float64 potential (1e-11 of the
maximum, the bound of the pinned potentials)."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("nx,ny,elements,slices,atoms", [(64, 48, 3, 9, 5), (100, 128, 25, 4, 60), (250, 331, 2, 3, 7),
                                                         (1024, 1024, 20, 2, 45)])
def test_against_float64(nx, ny, elements, slices, atoms):
    rng = np.random.default_rng(nx)
    box = (0.1 * nx, 0.1 * ny, 2.0 * slices)
    numbers = np.concatenate([np.arange(1, elements + 1), rng.integers(1, elements + 1, atoms - elements)])
    positions = rng.uniform(0, 1, (atoms, 3)) * box
    # all in the first and last slices where there are more than two: the others stay empty
    positions[:, 2] = np.where(rng.random(atoms) < 0.8, 1.0, 2.0 * slices - 0.5)
    ref = O.Potential.from_structure(O.Structure(box, numbers, positions), nx, ny, slice_thickness=2.0).build()
    got = sk.Potential(sk.AtomicStructure(box, numbers, positions), nx, ny, slice_thickness=2.0).build().values
    for a, b in zip(got, ref):
        assert np.abs(a - b).max() <= 1e-11 * max(np.abs(r).max() for r in ref)
    for j in range(1, slices - 1):
        assert not got[j].any()
