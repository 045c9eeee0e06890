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


@pytest.mark.parametrize("nn", [(128, 128, 128), (131, 127, 129), (200, 201, 203)])
def test_large_reads_fill_every_value(pic, nn):
    """Arrays whose pages are first written by several threads: shares of whole pages, an odd last one, and an
    output that the caller has already used and that does not start on a page."""
    W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    v = np.random.default_rng(0).normal(size=W.nv)
    W.phi = v
    got = W.phi
    assert np.max(np.abs(got - v)) <= 1e-13 * np.max(np.abs(v))  # float-float storage
    used = np.full(W.nv + 3, 7.0)
    out = used[1:-2]
    assert W._L.pic_world_get_field(W._h, 0, out.ctypes.data) == pic.PIC_OK
    assert np.array_equal(out, got) and used[0] == 7.0 and np.all(used[-2:] == 7.0)
    W.close()
