"""A call that returns host arrays cannot be part of a user's stream capture: it is refused, and the engine works on as
before once the capture has ended, on that stream and on its own."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sk = pytest.importorskip("simulatokit_b200")

RELAXED = 2  # cudaStreamCaptureModeRelaxed


@pytest.fixture()
def cudart():
    return ctypes.CDLL("libcudart.so.12")


@pytest.mark.parametrize("warm", [False, True])
def test_engine_after_a_refused_capture(cudart, warm):
    engine = sk.Engine(0)
    rng = np.random.default_rng(1)
    pot = sk.ProjectedPotential(sk.Grid(96, 96, 6.0, 6.0), rng.uniform(0, 20, (3, 96, 96)), [2.0] * 3)
    wave = sk.Waves.plane_wave(sk.ElectronBeam(200e3), pot.grid)
    ref = sk.Multislice.run(wave, pot, engine=sk.Engine(0))[-1].field
    if warm:
        assert np.array_equal(sk.Multislice.run(wave, pot, engine=engine)[-1].field, ref)
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cudart.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    engine.set_stream(stream.value)
    assert cudart.cudaStreamBeginCapture(stream, RELAXED) == 0
    with pytest.raises(sk.SimulatoError):
        sk.Multislice.run(wave, pot, engine=engine)
    cudart.cudaStreamEndCapture(stream, ctypes.byref(graph))
    if graph.value:
        assert cudart.cudaGraphDestroy(graph) == 0
    cudart.cudaGetLastError()
    assert np.array_equal(sk.Multislice.run(wave, pot, engine=engine)[-1].field, ref)
    engine.set_stream(None)
    assert np.array_equal(sk.Multislice.run(wave, pot, engine=engine)[-1].field, ref)
    assert cudart.cudaStreamDestroy(stream) == 0
