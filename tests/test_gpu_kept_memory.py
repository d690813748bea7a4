"""Memory that calls share: freed device blocks handed out again, and the pinned halves that waves go through. Batches
whose waves take less than one half, exactly one (2^20 points), and several with a remainder come back as each wave
alone does, bit for bit; potentials made and dropped in turn by two threads, each with a context of its own, give the
waves that the first of each gave."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


def _potential(n, slices, seed):
    rng = np.random.default_rng(seed)
    return sk.ProjectedPotential(sk.Grid(n, n, 0.06 * n, 0.06 * n), rng.uniform(0, 20, (slices, n, n)), [2.0] * slices)


@pytest.mark.parametrize("n,count", [(64, 3), (512, 4), (320, 23), (600, 7)])
def test_batches_through_the_halves(n, count):
    pot = _potential(n, 2, 1)
    beam = sk.ElectronBeam(200e3)
    rng = np.random.default_rng(2)
    waves = [sk.Waves(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)), pot.grid, beam) for _ in range(count)]
    together = sk.Multislice.runBatch(waves, pot)
    for k in (0, count // 2, count - 1):
        alone = sk.Multislice.run(waves[k], pot)[-1]
        assert np.array_equal(together[k].field, alone.field)


def test_blocks_between_threads():
    failures = []

    def work(seed):
        engine = sk.Engine(0)
        beam = sk.ElectronBeam(200e3)
        first = {}
        for turn in range(12):
            n = (96, 128, 100)[(turn + seed) % 3]
            pot = _potential(n, 3, seed)
            got = sk.Multislice.run(sk.Waves.plane_wave(beam, pot.grid), pot, engine=engine)[-1].field
            if not np.array_equal(first.setdefault(n, got), got):
                failures.append((seed, turn))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
