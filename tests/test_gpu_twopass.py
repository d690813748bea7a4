"""The two-pass engine (one shared-memory exchange a transform) at every length it takes, as rows and as columns, on
grids whose other side is another of its lengths (column counts that are not a multiple of its 8-column tiles among
them): a plane wave's exit wave, three probes' patterns and annular sums (an odd number of waves: the last group of a
block is short) against the float64 oracle. Bounds as the fused form's other tests: 1e-5 rel-L2 for waves, 1e-4 for
detector values."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")

LENGTHS = [128, 160, 192, 200, 240, 250, 256, 300, 320, 360, 384, 400, 450, 480, 500, 512, 576, 600, 640, 720, 750, 768,
           800, 900, 960, 1024]


@pytest.fixture(scope="module")
def engine():
    return sk.Engine.require()


@pytest.mark.parametrize("nx,ny", list(zip(LENGTHS, LENGTHS[7:] + LENGTHS[:7])))
def test_against_float64(engine, nx, ny):
    s = O.srtio3_cell().repeated(max(1, nx // 64), max(1, ny // 64), 1)
    op = O.Potential.from_structure(s, nx, ny, slice_thickness=1.9525)
    vs = op.build()
    ts = [O.transmission(v, 200e3, op.grid) for v in vs]
    wave = O.multislice(O.plane_wave(op.grid), ts, op.thicknesses, 200e3, op.grid)[-1]
    scan = sk.GridScan((0.3, 0.7), (3.905, 3.905), 3, 1)
    ores = O.stem_scan(O.ProbeSpec(200e3, 20.0), [(op.grid, vs, op.thicknesses)], scan.positions,
                       [O.DetectorSpec("annular", {"inner": 0, "outer": 20}),
                        O.DetectorSpec("annular", {"inner": 30, "outer": 70}),
                        O.DetectorSpec("pixelated", {"max_angle": "valid"})])
    pot = sk.Potential(sk.AtomicStructure(s.box, s.numbers, s.positions), nx, ny, slice_thickness=1.9525)
    ex = sk.Multislice.run(sk.Waves.plane_wave(sk.ElectronBeam(200e3), pot.grid), pot, engine=engine)[-1]
    assert O.rel_l2(ex.field, wave) <= 1e-5
    probe = sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0))
    dets = [sk.AnnularDetector(0, 20), sk.AnnularDetector(30, 70), sk.PixelatedDetector("valid")]
    for chosen in (dets, dets[:2]):  # with and without the k-space waves stored
        got = sk.STEM.scan(probe, [pot], scan, chosen, engine=engine)
        for m, r in zip(got, ores):
            assert O.rel_l2(m.values, np.asarray(r).ravel()) <= 1e-4
