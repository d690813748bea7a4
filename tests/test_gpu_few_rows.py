"""Rows of 512 points on either side of the row pass's rule for few of them (one row a warp up to four a multiprocessor, two
above): each wave of a batch above it has the bits of the wave alone, below it, for exit waves, job tables (a transmission a
wave) and scans, with row counts at the rule's edge and odd groups."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("nx,count", [(128, 5), (250, 3), (512, 2), (300, 2)])
def test_alone_and_together(nx, count):
    engine = sk.Engine.require()
    rng = np.random.default_rng(nx)
    grid = sk.Grid(nx, 512, 0.06 * nx, 0.06 * 512)
    beam = sk.ElectronBeam(200e3)
    pots = [sk.ProjectedPotential(grid, rng.uniform(0, 20, (3, nx, 512)), [2.0] * 3) for _ in range(count)]
    waves = [sk.Waves(rng.normal(size=(nx, 512)) + 1j * rng.normal(size=(nx, 512)), grid, beam) for _ in range(count)]
    together = sk.Multislice.runBatch(waves, pots[0], engine=engine)
    for w, t in zip(waves, together):
        assert np.array_equal(sk.Multislice.run(w, pots[0], engine=engine)[-1].field, t.field)
    tables = [sk.JobTable() for _ in range(count + 1)]
    for k, p in enumerate(pots):
        for t in (tables[0], tables[k + 1]):
            t.add_plane_wave(p, 200e3)
    for k, t in enumerate(tables[0].run(engine=engine)[0]):
        assert np.array_equal(tables[k + 1].run(engine=engine)[0][0], t)
    probe = sk.Probe(beam, grid, sk.Aperture(20.0))
    got = [sk.STEM.scan(probe, pots[:1], sk.GridScan((0, 0), (3, 3), count, 1), [sk.PixelatedDetector("valid")],
                        options=sk.ExecutionOptions(batch=b), engine=engine)[0].array() for b in (1, count)]
    assert np.array_equal(got[0], got[1])
