"""More detector sets than a context keeps plans of (64), scanned on one potential in batches whose slice loops are
captured and replayed: a plan made at the address of a dropped one must not meet the old plan's graph. Every image is the
one that launches without graphs give, bit for bit, over two rounds of the sets."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("n", [128, 250])
def test_seventy_annuli(n):
    engine = sk.Engine(0)
    rng = np.random.default_rng(n)
    pot = sk.ProjectedPotential(sk.Grid(n, n, 0.06 * n, 0.06 * n), rng.uniform(0, 20, (2, n, n)), [2.0] * 2)
    probe = sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0))
    scan = sk.GridScan((0, 0), (3, 3), 8, 1)
    sets = [[sk.AnnularDetector(0, 4 + 0.4 * k)] + [sk.AnnularDetector(20 + 0.4 * k, 60 + 2 * j) for j in range(k % 3)]
            for k in range(70)]
    images = {}
    for graphs in (False, True):
        options = sk.ExecutionOptions(batch=2, graphs=graphs)  # eager, captured, replayed twice
        for turn in range(2):
            for k, detectors in enumerate(sets):
                got = [m.array() for m in sk.STEM.scan(probe, [pot], scan, detectors, options=options, engine=engine)]
                assert all(np.array_equal(g, r) for g, r in zip(got, images.setdefault(k, got))), (graphs, turn, k)
