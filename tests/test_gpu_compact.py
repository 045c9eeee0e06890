"""Removal of the particles that leave: none, one, a few, most and all of them, at counts below and above a
CTA's and the grid's threads.  Exactly the ones whose straight path stays inside remain, unchanged by the
move into the holes, and the next pushes find them all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leave", [0.0, "one", 0.01, 0.5, 0.97, 1.0])
@pytest.mark.parametrize("n", [1, 300, 5_000, 400_000])
def test_survivors_are_kept_unchanged(pic, n, leave):
    nn = (17, 17, 17)
    W = pic.World(*nn, (0.0, 0.0, 0.0), (0.016, 0.016, 0.016))
    W.set_boundaries((0, 0, 0), (1,) * 6, (0.0,) * 6)
    e = pic.Species("e-", pic.ME, -pic.QE, W, 1.0, capacity=n + 1)
    rng = np.random.default_rng(n)
    gone = np.zeros(n, bool)
    if leave == "one":
        gone[rng.integers(n)] = True
    else:
        gone[rng.permutation(n)[:int(round(leave * n))]] = True
    pos = 0.004 + 0.008 * rng.random((n, 3))
    vel = np.zeros((n, 3))
    vel[gone, 2] = rng.choice([-1.0, 1.0], gone.sum()) * 4e7  # 0.02 m in a step; no field: the others stay
    w = 1.0 + rng.random(n)
    ids = rng.permutation(n).astype(np.uint64)
    e.addParticles(pos, vel, w, ids=ids, rewind=False)
    before = e.getPartRef()
    for _ in range(3):
        e.advance(5e-10, deposit=False)
        after = e.getPartRef()
        assert len(after) == n - gone.sum()
        keep = before[~np.isin(before["id"], ids[gone])]
        a, b = np.argsort(after["id"]), np.argsort(keep["id"])
        for f in ("id", "pos", "vel", "w"):
            assert np.array_equal(after[f][a], keep[f][b])
    W.close()
