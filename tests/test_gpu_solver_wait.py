"""A solve whose inner solver waits in vain leaves the potential as it was, and the next solve starts from it like a
solve without the failure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extrapolate", [False, True])
@pytest.mark.parametrize("method", ["rbsor", "pcg", "learned"])
@pytest.mark.parametrize("nn", [(21, 21, 21), (61, 60, 50)])  # one cluster, the whole GPU
def test_potential_is_unchanged(pic, nn, method, extrapolate):
    kind = dict(rbsor=pic.SOLVER_RBSOR, pcg=pic.SOLVER_PCG, learned=pic.SOLVER_LEARNED)[method]
    rho = np.random.default_rng(3).normal(size=int(np.prod(nn))) * 1e-6

    def solved(fail):
        W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
        W.set_boundaries((0, 0, 0), (1,) * 6, (0.0, 0.0, 0.0, 0.0, 0.0, 25.0))
        W.rho = rho
        S = pic.PotentialSolver(W, 20000, 1e-7, kind, omega=1.7)
        if extrapolate:
            S.setWarmStart(pic.WARM_EXTRAPOLATE)
        if fail:
            phi0 = W.phi
            assert W._L.pic_debug_set_wait_polls(W._h, 0) == pic.PIC_OK
            try:
                with pytest.raises(pic.PicError) as ei:
                    S.solve(raise_on_fail=True)
                assert ei.value.code == pic.PIC_ERR_DEVICE and "bounded wait" in str(ei.value)
            finally:
                assert W._L.pic_debug_set_wait_polls(W._h, -1) == pic.PIC_OK
            assert np.array_equal(W.phi, phi0)
        assert S.solve(raise_on_fail=True)
        phi, iters = W.phi, S.iters
        W.close()
        return phi, iters

    a, b = solved(True), solved(False)
    assert np.array_equal(a[0], b[0]) and a[1] == b[1]
