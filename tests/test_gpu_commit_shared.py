"""A push whose collisions, neutralisation and sputtering all append to one species counts every particle once:
the same push with a species for each gives as many, and the same ones."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import sigma_table

pytestmark = pytest.mark.gpu


def step(pic, shared):
    nn, xm, m = (17, 17, 17), (0.016, 0.016, 0.016), 16 * O.AMU
    W = pic.World(*nn, (0.0, 0.0, 0.0), xm)
    W.addBox((0.008, 0.008, 0.008), (0.006, 0.006, 0.006), 0.0)
    W.setTime(1e-10, 10)
    n = 40_000
    e = pic.Species("e-", pic.ME, -pic.QE, W, 10.0, capacity=3 * n)
    ion = pic.Species("O+", m, pic.QE, W, 10.0, capacity=3 * n)
    neu = ion if shared else pic.Species("O", m, pic.QE, W, 10.0, capacity=3 * n)
    spu = ion if shared else pic.Species("Sp", m, pic.QE, W, 10.0, capacity=3 * n)
    rng = np.random.default_rng(8)
    pos = rng.uniform(0.0, 0.016, (2 * n, 3)) * 0.999999
    pos = pos[~np.all(np.abs(pos - 0.008) <= 0.0031, axis=1)][:n]
    d = rng.normal(size=(n, 3))
    vel = np.sqrt(2 * rng.uniform(20, 300, n) * O.QE / O.ME)[:, None] * d / np.linalg.norm(d, axis=1)[:, None]
    e.addParticles(pos, vel, np.full(n, 10.0), ids=np.arange(n, dtype=np.uint64), rewind=False)
    E, S = sigma_table()
    M = pic.MC_MEX_Ionization(e, ion, W, 5e22, 300.0, m, 13.6, E, S, 0, (1.015e-18, 9.793, 61.81, 0.0), seed=77)
    e.set_object_interaction(1, neutrals=neu, spherium=spu, sputtering=True, seed=5)
    W.configure_loop(solve_each_step=False, sort_every=0)
    for _ in range(3):
        W.step()
    out = np.concatenate([s.getPartRef() for s in ([ion] if shared else [ion, neu, spu])])
    return np.sort(out, order=["id", "pos", "vel", "w"]), np.sort(e.getPartRef(), order="id"), M.stats(), e.object_stats()


def test_shared_species_is_committed_once(pic):
    a, ea, ma, oa = step(pic, True)
    b, eb, mb, ob = step(pic, False)
    assert mb["ionizations"] and ob["impacts"]  # all three kinds of append occur
    assert ma == mb and oa == ob and len(ea) == len(eb) and len(a) == len(b)
    assert np.array_equal(ea["id"], eb["id"]) and np.array_equal(a["id"], b["id"])
