"""Conservation sums and field energy at counts around the runs of a thread, a CTA and the grid, against FP64
numpy sums.  The device sums are compensated FP32 per thread and FP64 above: 1e-12 of the sum of absolute
values covers the exact terms' 2^-47; |v|^2 is rounded to FP32 once (3 roundings: 2e-7)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 8192, 8193, 100_003, 3_000_000])
def test_sums_match_fp64(pic, n):
    W = pic.World(9, 9, 9, (0.0, 0.0, 0.0), (0.008, 0.008, 0.008))
    e = pic.Species("e-", pic.ME, -pic.QE, W, 1.0, capacity=max(n, 1))
    rng = np.random.default_rng(n)
    if n:
        e.addParticles(0.001 + 0.006 * rng.random((n, 3)), rng.normal(1e5, 1e6, (n, 3)),
                       rng.lognormal(3.0, 0.5, n), rewind=False)
    p = e.getPartRef()
    v, w = p["vel"], p["w"]  # the FP32 values, exact in FP64
    s = e.sums()
    assert abs(s[0] - w.sum()) <= 1e-12 * w.sum()
    for d in range(3):
        assert abs(s[1 + d] - pic.ME * (w * v[:, d]).sum()) <= 1e-12 * pic.ME * np.abs(w * v[:, d]).sum()
    ke = 0.5 * pic.ME * (w * (v * v).sum(1)).sum()
    assert abs(s[4] - ke) <= 2e-7 * ke
    assert np.array_equal(e.sums(), s)  # the order of the additions is fixed
    W.close()


@pytest.mark.parametrize("nn,per", [((2, 2, 2), (0, 0, 0)), ((5, 7, 9), (1, 1, 0)), ((33, 29, 41), (0, 0, 0)),
                                    ((64, 65, 130), (1, 0, 1)), ((129, 128, 97), (1, 1, 1))])
def test_field_energy_matches_fp64(pic, nn, per):
    xm = np.array([1e-3 * (n - 1) for n in nn])
    W = pic.World(*nn, (0.0, 0.0, 0.0), xm)
    W.set_boundaries(per, (1,) * 6, (0.0,) * 6)
    W.ef = np.random.default_rng(1).normal(0.0, 100.0, (W.nv, 3))
    E = np.asarray(W.ef).reshape(nn[2], nn[1], nn[0], 3).astype(np.float32).astype(np.float64)
    vol = np.ones(nn[::-1])
    for d in range(3):
        first, last = [slice(None)] * 3, [slice(None)] * 3
        first[2 - d], last[2 - d] = 0, nn[d] - 1
        if per[d]:
            vol[tuple(last)] = 0.0
        else:
            vol[tuple(first)] *= 0.5
            vol[tuple(last)] *= 0.5
    ref = 0.5 * 8.85418782e-12 * 1e-9 * ((E ** 2).sum(-1) * vol).sum()
    assert abs(W.getPE() - ref) <= 1e-9 * ref
    W.close()
