"""The Poisson inner solvers that keep a whole grid on the chip: one thread-block cluster for small
grids, a persistent kernel over the whole GPU for mid-size ones.  Every geometry rule that they restate
(halo planes, rings, seams of periodic axes with an odd number of nodes, mirror walls, objects, thin and
one-plane slabs, rows of every remainder by four, short rows, the largest grids of each register form) is solved and compared with the FP64 oracle's converged answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    # nn, periodic, walls fixed (else mirror), boxes (centre, sides, volts) in units of the box
    "walls_21": ((21, 21, 21), (0, 0, 0), 1, ()),
    "two_cells": ((5, 3, 3), (0, 0, 0), 1, ()),
    "one_inner_plane": ((33, 29, 3), (0, 0, 0), 1, ()),
    "xy_periodic_even": ((17, 9, 30), (1, 1, 0), 1, ()),
    "xy_seams": ((16, 10, 35), (1, 1, 0), 1, ()),
    "ring_all_seams": ((16, 18, 20), (1, 1, 1), 1, (((0.5, 0.5, 0.5), (0.3, 0.3, 0.3), 40.0),)),
    "ring_one_plane_each": ((12, 14, 17), (0, 0, 1), 1, ()),
    "mirror_walls_box": ((19, 15, 23), (0, 0, 0), 0, (((0.5, 0.5, 0.0), (2.0, 2.0, 0.2), 100.0),)),
    "widest_planes": ((60, 61, 40), (0, 0, 0), 1, ()),
    "above_one_cluster": ((67, 66, 45), (1, 0, 0), 1, ()),
    "rows_of_64": ((64, 60, 50), (1, 1, 0), 1, ()),
    "rows_of_62_mirror": ((62, 61, 44), (0, 1, 0), 0, (((0.5, 0.5, 0.0), (2.0, 2.0, 0.1), 30.0),)),
    "short_rows": ((3, 5, 8000), (0, 0, 0), 1, ()),
    "ring_of_the_grid": ((57, 55, 60), (1, 1, 1), 1, (((0.4, 0.5, 0.5), (0.2, 0.3, 0.3), 40.0),)),
}


def setup(pic, port, name):
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
    return W, g, kind


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("method", ["rbsor", "pcg"])
def test_converges_to_the_oracles_answer(pic, port, name, method):
    W, g, kind = setup(pic, port, name)
    phi0 = W.phi
    S = pic.PotentialSolver(W, 20000, 1e-9, pic.SOLVER_RBSOR if method == "rbsor" else pic.SOLVER_PCG, omega=1.7)
    assert S.solve(raise_on_fail=True) and S.rel <= 1e-9
    phi, rho = W.phi, W.rho
    ref = phi0.copy()
    assert port.solve_fpcg(g, kind, ref, rho, 1e-13, 20000)[0]
    # the device's own stopping rule, measured in FP64 (the float-float residual is good to 1e-13)
    assert port.rel_residual(g, kind, phi, rho) <= 2e-9
    assert np.max(np.abs(phi - ref)) <= 1e-6 * np.max(np.abs(ref))
    # the same solve again is the same to the last bit: no sum or sweep depends on timing
    W.phi = phi0
    assert S.solve(raise_on_fail=True)
    assert np.array_equal(W.phi, phi)
    W.close()


@pytest.mark.parametrize("name", ["walls_21", "ring_all_seams", "rows_of_64"])
@pytest.mark.parametrize("method", ["rbsor", "pcg"])
def test_wait_that_runs_out_is_reported_and_solver_recovers(pic, port, name, method):
    W, g, kind = setup(pic, port, name)
    phi0 = W.phi
    S = pic.PotentialSolver(W, 20000, 1e-9, pic.SOLVER_RBSOR if method == "rbsor" else pic.SOLVER_PCG, omega=1.7)
    assert W._L.pic_debug_set_wait_polls(W._h, 0) == pic.PIC_OK
    try:
        with pytest.raises(pic.PicError) as ei:
            S.solve(raise_on_fail=True)
        assert ei.value.code == pic.PIC_ERR_DEVICE and "bounded wait" in str(ei.value)
    finally:
        assert W._L.pic_debug_set_wait_polls(W._h, -1) == pic.PIC_OK
    W.phi = phi0
    assert S.solve(raise_on_fail=True)
    assert port.rel_residual(g, kind, W.phi, W.rho) <= 2e-9
    W.close()
