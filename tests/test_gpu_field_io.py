"""Node fields to and from the caller's FP64 arrays: the conversions run on the device through a
staging buffer, so a round trip is compared exactly with the same conversions in numpy, on a grid that
fits one staging round and on one that needs several (with a remainder)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nn", [(5, 7, 3), (161, 163, 165)])  # 4.33 M nodes: rounds of 4194304 doubles
def test_field_round_trip_is_exact(pic, nn):
    W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    rng = np.random.default_rng(3)
    a = rng.normal(size=W.nv) * 10.0 ** rng.integers(-12, 12, W.nv)
    a[:4] = [0.0, -0.0, 1e-320, 3.4e38]
    W.phi = a
    hi = a.astype(np.float32)
    lo = (a - hi.astype(np.float64)).astype(np.float32)
    assert np.array_equal(W.phi, hi.astype(np.float64) + lo.astype(np.float64))
    W.rho = a
    assert np.array_equal(W.rho, hi.astype(np.float64))
    e = rng.normal(size=(W.nv, 3))
    W.ef = e
    assert np.array_equal(W.ef, e.astype(np.float32).astype(np.float64))
    W.close()
