"""The finest level of the learned preconditioner on grids large enough for the kernel that marches along z:
odd and even counts, seams and walls on every axis, columns that end inside the box, shares that cross from
one column to the next, against the FP64 numpy restatement; and through a solve, whose sums it forms."""
import numpy as np
import pytest

import learned_ref as LR
from test_gpu_learned import distinct, free_mask, unpack

pytestmark = pytest.mark.gpu

GEOMS = {
    "seams_xy_odd": ((132, 35, 701), (1, 1, 0)),      # 131 x 34 distinct nodes
    "seam_z_odd": ((68, 50, 1002), (0, 0, 1)),        # 1001 distinct planes
    "walls": ((64, 33, 1700), (0, 0, 0)),             # one column in x, a row past the second in y
    "seams_all": ((72, 81, 513), (1, 1, 1)),
}


@pytest.mark.parametrize("geom", sorted(GEOMS))
def test_apply_matches_oracle(pic, geom):
    nn, per = GEOMS[geom]
    g = dict(nn=nn, per=per, xm=tuple(1e-3 * (n - 1) * s for n, s in zip(nn, (1.0, 1.2, 0.9))))
    W = pic.World(*nn, (0.0, 0.0, 0.0), g["xm"])
    W.set_boundaries(per, (1,) * 6, (0.0,) * 6)
    lp = pic.LearnedPreconditioner(W)
    rng = np.random.default_rng(11)
    w0 = lp.weights()
    w = w0 + rng.normal(size=w0.size).astype(np.float32) * np.float32(0.2) * np.abs(w0).max()
    lp.set_weights(w)
    r = rng.normal(size=int(np.prod(nn)))
    z = lp.apply(r)
    _, diag = lp.levels()
    ref = LR.apply(distinct(r, g), free_mask(g), unpack(w), tuple(bool(p) for p in per[::-1]), diag)
    # the bound of the other hierarchies' tests: FP32 sums of 125 taps over the levels
    assert np.max(np.abs(distinct(z, g) - ref)) <= 2e-5 * np.max(np.abs(ref))
    full = np.zeros(r.size, bool)
    full[distinct(np.arange(r.size), g).ravel()[free_mask(g).ravel() > 0]] = True
    assert np.all(z[~full] == 0)
    assert np.array_equal(lp.apply(r), z)
    if all(per):
        W.close()  # without a fixed node the Poisson problem is singular
        return
    # the solve uses the sums z.r and z.q: it converges as the other forms' solves do
    W.rho = 1e-7 * r
    S = pic.PotentialSolver(W, 200, 1e-6, pic.SOLVER_LEARNED)
    lp.set_weights(w0)
    assert S.solve(raise_on_fail=True) and S.rel <= 1e-6
    W.close()
