"""The two column engines that the fused form has at 256, 512 and 1024, by SIMK_OPT_COL_TILE: 0 names the two-pass kernels, 4
the register engine (one column a thread). Other kernels, so the waves differ in their last bits; they agree to 1e-6
(waves, patterns and annular sums), each is within 1e-6 of the float64 oracle's exit wave, and one engine used with both
values in turn, eagerly and from graphs, gives each time the bits of the value asked for; a job table likewise."""

import numpy as np
import pytest

from oracle import simk_oracle as O

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


@pytest.mark.parametrize("nx,ny", [(256, 256), (512, 200), (1024, 256)])
def test_two_pass_and_register_columns(nx, ny):
    engine = sk.Engine.require()
    rng = np.random.default_rng(nx)
    grid = O.Grid(nx, ny, 0.06 * nx, 0.06 * ny)
    values = rng.uniform(0, 20, (3, nx, ny))
    ref = O.multislice(O.plane_wave(grid), [O.transmission(v, 200e3, grid) for v in values], [2.0] * 3, 200e3, grid)[-1]
    pot = sk.ProjectedPotential(sk.Grid(nx, ny, 0.06 * nx, 0.06 * ny), values, [2.0] * 3)
    probe = sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0))
    scan = sk.GridScan((0, 0), (3, 3), 6, 1)
    table = sk.JobTable()
    table.add_plane_wave(pot, 200e3)
    table.add_probe(pot, probe, (1.0, 2.0))
    first = {}
    for turn in range(3):
        for tile in (0, 4):
            options = sk.ExecutionOptions(batch=2, col_tile=tile)
            wave = sk.Multislice.run(sk.Waves.plane_wave(probe.beam, pot.grid), pot, options=options, engine=engine)
            scans = sk.STEM.scan(probe, [pot], scan, [sk.AnnularDetector(0, 20), sk.PixelatedDetector("valid")],
                                 options=options, engine=engine)
            got = [wave[-1].field] + [m.array() for m in scans] + list(table.run(options=options, engine=engine)[0])
            for a, b in zip(first.setdefault(tile, got), got):
                assert np.array_equal(a, b)
    assert not np.array_equal(first[0][0], first[4][0])
    for a, b in zip(first[0], first[4]):
        assert O.rel_l2(a, b) <= 1e-6
    for tile in (0, 4):
        assert O.rel_l2(first[tile][0], ref) <= 1e-6
