"""SOR sweeps on one thread-block cluster where a CTA sends its neighbours nothing in some or all passes: a plate
across the box at a slab's first plane with unequal compartments on its sides, a last slab that is a fixed wall plane
alone, a ring in z only with an odd number of planes (its last plane is relaxed in passes of its own) and a last
slab of one plane.  Compared with the FP64 oracle's converged answer, and every repetition to the last bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # nn, periodic, planes of a CTA, boxes (centre, sides, volts) in units of the box
    "plate_at_a_slab": ((21, 21, 33), (0, 0, 0), 3, (((0.5, 0.5, 15 / 32), (2.0, 2.0, 0.01), 40.0),
                                                     ((0.5, 0.5, 0.8), (0.8, 0.8, 0.3), -10.0))),
    "plate_wide_slabs": ((45, 45, 48), (0, 0, 0), 3, (((0.5, 0.5, 24 / 47), (2.0, 2.0, 0.01), 40.0),
                                                      ((0.5, 0.5, 0.3), (0.9, 0.9, 0.2), -10.0))),
    "wall_plane_alone": ((21, 21, 21), (0, 0, 0), 2, ()),
    "wall_plane_beside_wide_slabs": ((55, 55, 31), (0, 0, 0), 2, ()),
    "z_seam_alone": ((21, 19, 32), (0, 0, 1), 2, ()),
    "z_seam_beside_wide_slabs": ((55, 55, 32), (0, 0, 1), 2, (((0.3, 0.5, 0.2), (0.2, 0.4, 0.1), 15.0),)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_converges_and_repeats_to_the_last_bit(pic, port, name):
    nn, per, planes, boxes = CASES[name]
    stack = nn[2] - per[2]
    assert planes == -(-stack // 16) and planes * nn[0] * nn[1] <= 6144  # the one-cluster form takes it
    L = 1e-3 * (np.array(nn) - 1) * np.array([1.0, 1.3, 0.8])
    bx = [(np.array(c) * L, np.array(s) * L, v) for c, s, v in boxes]
    g = port.grid(nn, (0, 0, 0), L, periodic=per, boxes=[(c, s) for c, s, _ in bx])
    kind = port.node_kinds(g, 1)
    W = pic.World(*nn, (0.0, 0.0, 0.0), L)
    W.set_boundaries(per, (1,) * 6, (0.0, 0.0, 0.0, 0.0, 0.0, 0.0 if per[2] else 25.0))
    for c, s, v in bx:
        W.addBox(c, s, v)
    W.rho = np.random.default_rng(5).normal(size=W.nv) * 1e-5 + 2e-6
    phi0 = W.phi
    S = pic.PotentialSolver(W, 20000, 1e-9, pic.SOLVER_RBSOR, omega=1.7)
    assert S.solve(raise_on_fail=True) and S.rel <= 1e-9
    phi = W.phi
    ref = phi0.copy()
    assert port.solve_fpcg(g, kind, ref, W.rho, 1e-13, 20000)[0]
    assert port.rel_residual(g, kind, phi, W.rho) <= 2e-9
    assert np.max(np.abs(phi - ref)) <= 1e-6 * np.max(np.abs(ref))
    for _ in range(10):
        W.phi = phi0
        assert S.solve(raise_on_fail=True)
        assert np.array_equal(W.phi, phi)
    W.close()
