"""The two-pass column kernel's ring of tile buffers at every length it takes: so many waves that every block fills each of
its buffers at least three times, a count that leaves the last group of waves short, through the probes' generation, the
slices' passes and the last pass with the detectors in its epilogue, with the waves stored beside them, and without
(modes 2, 0, 3 and 1). Each wave is the one that batches of one wave (one buffer a block, never refilled) give, bit for
bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")

LENGTHS = [160, 192, 200, 240, 250, 256, 300, 320, 360, 384, 400, 450, 480, 500, 512, 576, 600, 640, 720, 750, 768, 800,
           900, 960, 1024]
SMS, COLUMNS = 148, 64


@pytest.mark.parametrize("n", LENGTHS)
def test_bits_of_single_waves(n):
    buffers = (222 * 1024 - 16 * n) // (64 * n)
    count = -(-3 * buffers * SMS // (COLUMNS // 8)) + 1
    engine = sk.Engine.require()
    rng = np.random.default_rng(n)
    pot = sk.ProjectedPotential(sk.Grid(n, COLUMNS, 0.06 * n, 0.06 * COLUMNS), rng.uniform(0, 20, (2, n, COLUMNS)),
                                [2.0] * 2)
    probe = sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0))
    scan = sk.GridScan((0, 0), (3, 3), count, 1)
    annular = [sk.AnnularDetector(0, 20), sk.AnnularDetector(30, 90)]
    for detectors, epilogue in ((annular, True), (annular + [sk.PixelatedDetector("valid")], True), (annular, False)):
        got = {}
        for batch in (1, count):
            options = sk.ExecutionOptions(batch=batch, epilogue_detect=epilogue)
            got[batch] = [m.array() for m in sk.STEM.scan(probe, [pot], scan, detectors, options=options, engine=engine)]
        for one, all_ in zip(got[1], got[count]):
            assert np.array_equal(one, all_)
