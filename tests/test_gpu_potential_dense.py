"""Groups of atoms on either side of the builder's rule for merging their weights (sorted up to N / 8 atoms, in a dense
image above), in one build: at the rule, one more, many atoms a pixel, and a slice of few beside one of many, against the
oracle's float64 potential (1e-11 of the maximum, the bound of the pinned potentials)."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("nx,ny,counts", [(40, 36, (180, 181)), (40, 36, (181, 180, 3)), (16, 16, (4000, 1, 33)),
                                          (128, 96, (1536, 1537, 9000))])
def test_against_float64(nx, ny, counts):
    rng = np.random.default_rng(nx)
    box = (0.2 * nx, 0.2 * ny, 2.0 * len(counts))
    atoms = sum(counts)
    positions = rng.uniform(0, 1, (atoms, 3)) * box
    positions[:, 2] = np.repeat(2.0 * np.arange(len(counts)) + 1.0, counts)
    for numbers in (np.full(atoms, 14), rng.integers(13, 16, atoms)):
        ref = O.Potential.from_structure(O.Structure(box, numbers, positions), nx, ny, slice_thickness=2.0).build()
        got = sk.Potential(sk.AtomicStructure(box, numbers, positions), nx, ny, slice_thickness=2.0).build().values
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= 1e-11 * max(np.abs(r).max() for r in ref)
