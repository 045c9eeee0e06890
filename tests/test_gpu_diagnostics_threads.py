"""Conservation sums and the field energy asked for by other host threads while one thread solves: every solve takes
the same iterations to the same potential as alone, and every diagnostic gives its own value."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_diagnostics_during_solves(pic):
    W = pic.World(21, 21, 21, (0.0, 0.0, 0.0), (0.02, 0.02, 0.02))
    W.set_boundaries((0, 0, 0), (1,) * 6, (0.0,) * 6)
    rng = np.random.default_rng(1)
    s = pic.Species("e-", pic.ME, -pic.QE, W, 1.0, capacity=20_000)
    s.addParticles(0.001 + 0.018 * rng.random((20_000, 3)), rng.normal(0, 1e6, (20_000, 3)), np.full(20_000, 3.0),
                   rewind=False)
    W.rho = rng.normal(size=W.nv) * 1e-6
    W.ef = rng.normal(size=(W.nv, 3))
    phi0 = W.phi
    S = pic.PotentialSolver(W, 5000, 1e-8, pic.SOLVER_PCG)
    assert S.solve(raise_on_fail=True)
    phi, iters, sums, pe = W.phi, S.iters, s.sums(), W.getPE()
    stop, wrong, count = threading.Event(), [], [0, 0]

    def ask(k, f, ref):
        try:
            while not stop.is_set():
                v = f()
                count[k] += 1
                if not np.array_equal(v, ref):
                    wrong.append((k, v))
        except Exception as e:  # reported by the assertion below
            wrong.append(e)

    threads = [threading.Thread(target=ask, args=(0, s.sums, sums)), threading.Thread(target=ask, args=(1, W.getPE, pe))]
    for t in threads:
        t.start()
    try:
        for _ in range(300):
            W.phi = phi0
            assert S.solve(raise_on_fail=True) and S.iters == iters
            assert np.array_equal(W.phi, phi)
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not wrong and min(count) > 0
    W.close()
