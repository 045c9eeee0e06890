"""Learned preconditioner on hierarchies whose levels take every form of the apply: tiled kernels above
the coarse part, coarse levels spread over the GPU with 1 to 32 lanes per voxel, and the redundant levels
in shared memory, on odd, periodic, thin and long boxes, against the FP64 numpy restatement."""
import numpy as np
import pytest

import learned_ref as LR
from test_gpu_learned import coeffs, distinct, free_mask, unpack

pytestmark = pytest.mark.gpu

GEOMS = {
    "first_level_joins": dict(nn=(65, 65, 127), per=(1, 1, 0)),      # level 1: 65 536 voxels
    "second_level_joins": dict(nn=(97, 81, 131), per=(1, 1, 0)),     # level 1: 126 720, level 2: 15 840
    "dirichlet_odd": dict(nn=(67, 71, 69), per=(0, 0, 0)),
    "ring_odd": dict(nn=(52, 40, 38), per=(1, 1, 1)),
    "thin": dict(nn=(5, 6, 3000), per=(0, 1, 0)),
    "all_redundant": dict(nn=(20, 17, 33), per=(1, 0, 0)),
}


@pytest.mark.parametrize("geom", sorted(GEOMS))
def test_apply_matches_oracle_on_every_level_form(pic, geom):
    nn, per = GEOMS[geom]["nn"], GEOMS[geom]["per"]
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
    # the bound of the small hierarchies' test: FP32 sums of 125 taps over the levels
    assert np.max(np.abs(distinct(z, g) - ref)) <= 2e-5 * np.max(np.abs(ref))
    assert np.array_equal(lp.apply(r), z)  # the same bits again: the order of the sums is fixed
    W.close()


def test_wait_that_runs_out_is_reported_and_the_preconditioner_recovers(pic):
    nn = GEOMS["second_level_joins"]["nn"]
    W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    W.set_boundaries((1, 1, 0), (1,) * 6, (0.0,) * 6)
    lp = pic.LearnedPreconditioner(W)
    r = np.random.default_rng(2).normal(size=W.nv)
    z = lp.apply(r)
    S = pic.PotentialSolver(W, 2000, 1e-6, pic.SOLVER_LEARNED)
    W.rho = r * 1e-7
    assert W._L.pic_debug_set_wait_polls(W._h, 0) == pic.PIC_OK
    try:
        for call in (lambda: lp.apply(r), lambda: S.solve(raise_on_fail=True)):
            with pytest.raises(pic.PicError) as ei:
                call()
            assert ei.value.code == pic.PIC_ERR_DEVICE and "bounded wait" in str(ei.value)
    finally:
        assert W._L.pic_debug_set_wait_polls(W._h, -1) == pic.PIC_OK
    assert np.array_equal(lp.apply(r), z)
    assert S.solve(raise_on_fail=True)
    W.close()
