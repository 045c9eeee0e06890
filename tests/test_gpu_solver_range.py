"""Inner CG solves whose sums leave FP32's range although no node's share does: the same charge times a power of two
takes the same iterations to the same potential times that power."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["pcg", "learned"])
@pytest.mark.parametrize("nn", [(21, 21, 21), (45, 45, 45), (64, 64, 60), (129, 65, 97)])  # cluster, cluster, GPU, GPU
def test_amplitude_is_a_factor(pic, nn, method):
    kind = pic.SOLVER_PCG if method == "pcg" else pic.SOLVER_LEARNED
    rho = np.random.default_rng(3).normal(size=int(np.prod(nn))).astype(np.float32) * np.float32(2.0 ** -20)
    ref = None
    for power in (0, 40, -40):  # rho of 1e-6, 1e6 and 1e-18 C/m^3: |r|^2 of up to 1e40 at 1e6
        W = pic.World(*nn, (0.0, 0.0, 0.0), tuple(1e-3 * (n - 1) for n in nn))
        W.set_boundaries((0, 0, 0), (1,) * 6, (0.0,) * 6)
        W.rho = rho * 2.0 ** power
        S = pic.PotentialSolver(W, 20000, 1e-8, kind)
        assert S.solve(raise_on_fail=True)
        phi, iters = W.phi * 2.0 ** -power, S.iters
        W.close()
        if ref is None:
            ref = phi, iters
        assert iters == ref[1] and np.array_equal(phi, ref[0])


def test_thin_box_of_many_tiles(pic):
    """A grid whose 32 x 8 x 8 tiles are mostly empty: a CTA of the persistent learned CG owns more tiles than a thread
    sums in FP32 at once."""
    nn = (33, 9, 4000)  # 2 x 2 x 500 tiles, 13 or 14 for a CTA
    W = pic.World(*nn, (0.0, 0.0, 0.0), tuple(1e-3 * (n - 1) for n in nn))
    W.set_boundaries((0, 0, 0), (1,) * 6, (0.0,) * 6)
    W.rho = np.random.default_rng(3).normal(size=W.nv) * 1e-6
    phi0 = W.phi
    phi = []
    for kind in (pic.SOLVER_LEARNED, pic.SOLVER_PCG):
        W.phi = phi0
        S = pic.PotentialSolver(W, 20000, 1e-9, kind)
        assert S.solve(raise_on_fail=True) and S.rel <= 1e-9
        phi.append(W.phi)
    # two residuals of 1e-9 through the condition number, 4 (8^2 / pi^2) x 3 axes at most
    assert np.max(np.abs(phi[0] - phi[1])) <= 2e-9 * 80 * np.max(np.abs(phi[1]))
    W.close()
