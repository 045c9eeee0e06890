"""Solves with the learned preconditioner that run as one persistent kernel over the GPU: grids of one
partial tile, of several tiles per SM, with seams of periodic axes, mirror walls, objects, and with no,
one or more levels between the fine grid and the dense coarse operator, against the FP64 oracle's
converged answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # nn, periodic, walls fixed (else mirror), boxes (centre, sides, volts) in units of the box
    "dense_level_1": ((17, 17, 19), (1, 1, 0), 1, ()),            # 8 x 8 x 9 voxels: no level between
    "dense_level_2": ((31, 31, 51), (0, 0, 0), 1, ()),            # level 1: 5850 voxels
    "edges_of_a_tile": ((33, 9, 9), (0, 0, 0), 1, ()),
    "seams": ((32, 40, 38), (1, 1, 1), 1, (((0.5, 0.5, 0.5), (0.3, 0.3, 0.3), 40.0),)),
    "mirror_box": ((35, 30, 27), (0, 0, 0), 0, (((0.5, 0.5, 0.0), (2.0, 2.0, 0.2), 100.0),)),
    "long": ((5, 6, 3000), (0, 1, 0), 1, ()),
    "tiles_in_turn": ((97, 81, 131), (1, 1, 0), 1, ()),           # 1.0 M nodes, 6 tiles per SM at most
    "ragged_tiles": ((129, 65, 120), (1, 0, 0), 1, (((0.4, 0.5, 0.5), (0.2, 0.3, 0.3), 40.0),)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_converges_to_the_oracles_answer(pic, port, name):
    nn, per, fixed, boxes = CASES[name]
    L = 1e-3 * (np.array(nn) - 1) * np.array([1.0, 1.3, 0.8])
    bx = [(np.array(c) * L, np.array(s) * L, v) for c, s, v in boxes]
    g = port.grid(nn, (0, 0, 0), L, periodic=per, boxes=[(c, s) for c, s, _ in bx])
    kind = port.node_kinds(g, fixed)
    W = pic.World(*nn, (0.0, 0.0, 0.0), L)
    W.set_boundaries(per, (fixed,) * 6, (0.0, 0.0, 0.0, 0.0, 0.0, 25.0 if not per[2] else 0.0))
    for c, s, v in bx:
        W.addBox(c, s, v)
    W.rho = np.random.default_rng(5).normal(size=W.nv) * 1e-5 + 2e-6
    phi0 = W.phi
    S = pic.PotentialSolver(W, 5000, 1e-9, pic.SOLVER_LEARNED)
    assert S.solve(raise_on_fail=True) and S.rel <= 1e-9
    phi, rho = W.phi, W.rho
    ref = phi0.copy()
    assert port.solve_fpcg(g, kind, ref, rho, 1e-13, 20000)[0]
    # the bounds of the other inner solvers' test: the stopping rule in FP64, and the answer
    assert port.rel_residual(g, kind, phi, rho) <= 2e-9
    assert np.max(np.abs(phi - ref)) <= 1e-6 * np.max(np.abs(ref))
    # the same solve again is the same to the last bit: no sum depends on timing
    W.phi = phi0
    assert S.solve(raise_on_fail=True)
    assert np.array_equal(W.phi, phi)
    W.close()
