"""Node fields, densities and gas properties on a device whose memory is used up: the conversions go through
the little staging that a world always has, and give the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(pic, nn):
    W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    s = pic.Species("O", 16 * pic.AMU, 0.0, W, 1e3, capacity=50_000)
    s.loadUniform((0, 0, 0), (1, 1, 1), 50_000, 300.0, 1e3, 0.0, seed=3)
    s.advance(1e-9, deposit=True)
    W.computeChargeDensity()
    s.updateAverages()
    s.sampleMoments()
    return W, s


def write(W):
    rng = np.random.default_rng(2)
    W.phi, W.rho, W.ef = rng.normal(size=W.nv), rng.normal(size=W.nv), rng.normal(size=(W.nv, 3))


def read(W, s):
    return [W.phi, W.rho, W.ef, s.den, s.den_avg, *s.computeGasProperties()]


def test_fields_without_device_memory(pic):
    torch = pytest.importorskip("torch")
    small, ss = make(pic, (9, 9, 9))  # every kernel of the test has run once: their code is loaded
    write(small)
    read(small, ss)
    W, s = make(pic, (97, 99, 101))  # 7.8 MB of potential, no field of it moved yet
    held = []
    try:
        for size in (1 << 32, 1 << 28, 1 << 21, 1 << 20):  # the last in segments of 2 MB
            while True:
                try:
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                except torch.OutOfMemoryError:
                    break
        write(W)
        short = read(W, s)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    for a, b in zip(short, read(W, s)):
        assert np.array_equal(a, b)
    write(W)
    for a, b in zip(short, read(W, s)):
        assert np.array_equal(a, b)
    W.close()
    small.close()
