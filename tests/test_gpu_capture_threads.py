"""Buffers are released in one thread while another captures its slice loops: each thread makes and drops potentials on a
context of its own, with scans whose slice loops are captured anew for every potential. The images are the ones of the
same scans alone, bit for bit."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")


def _scan(engine, n, seed):
    rng = np.random.default_rng(seed)
    pot = sk.ProjectedPotential(sk.Grid(n, n, 0.06 * n, 0.06 * n), rng.uniform(0, 20, (6, n, n)), [2.0] * 6)
    probe = sk.Probe(sk.ElectronBeam(200e3), pot.grid, sk.Aperture(20.0))
    scan = sk.GridScan((0, 0), (3, 3), 12, 1)
    options = sk.ExecutionOptions(batch=4)  # three batches: eager, captured, replayed
    got = sk.STEM.scan(probe, [pot], scan, [sk.AnnularDetector(0, 20)], options=options, engine=engine)
    return got[0].array()


@pytest.mark.parametrize("n", [96, 256])
def test_release_during_capture(n):
    engine = sk.Engine(0)
    alone = {seed: _scan(engine, n, seed) for seed in range(4)}
    failures = []

    def work(shift):
        mine = sk.Engine(0)
        for turn in range(16):
            seed = (turn + shift) % 4
            try:
                if not np.array_equal(_scan(mine, n, seed), alone[seed]):
                    failures.append((shift, turn))
            except Exception as e:  # a capture broken off by the other thread
                failures.append((shift, turn, str(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in (0, 1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
