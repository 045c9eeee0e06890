"""The push at the edges of its chunks and windows: counts around a chunk's size, particles in cell order,
scattered over the whole grid, in one cell, thinly spread and with weights far above the mean, against the
FP64 oracle with the tolerances of the parity tests."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import by_id, oracle_parts, smooth_field

pytestmark = pytest.mark.gpu

NN, PER = (37, 23, 45), (1, 1, 0)
XM = (0.036, 0.022, 0.044)


@pytest.mark.parametrize("order", ["cells", "random", "one_cell", "heavy"])
@pytest.mark.parametrize("n", [1, 511, 512, 513, 1537, 60_000, 700_000])
def test_push_and_deposit_match_the_oracle(pic, port, n, order):
    rng = np.random.default_rng(n + len(order))
    pos = rng.uniform(0.0, 1.0, (n, 3)) * XM * (1, 1, 0.98) + (0, 0, 0.01 * XM[2])
    if order == "one_cell":
        pos = (np.array((11, 7, 20)) + 0.05 + 0.9 * rng.uniform(size=(n, 3))) * 1e-3
    elif order != "random":
        c = np.floor(pos / 1e-3).astype(int)
        pos = pos[np.lexsort((c[:, 0], c[:, 1], c[:, 2]))]
    vel = rng.normal(0.0, 4e5, (n, 3))  # 0.3 cells a step on each axis
    w = rng.lognormal(0.0, 0.5, n) * 64.0
    if order == "heavy":
        w[rng.random(n) < 0.05] *= 1e4
    dt = 8e-10
    ef = smooth_field(int(np.prod(NN)), NN, None, 50.0, 3)
    W = pic.World(*NN, (0.0, 0.0, 0.0), XM)
    W.set_boundaries(PER, (1,) * 6, (0.0,) * 6)
    W.ef = ef
    e = pic.Species("e-", pic.ME, -pic.QE, W, 64.0, capacity=n + 16)
    ids = np.arange(n, dtype=np.uint64)
    e.addParticles(pos, vel, w, ids=ids, rewind=False)
    e.advance(dt, deposit=True)
    W.computeChargeDensity()
    g = port.grid(NN, (0.0, 0.0, 0.0), XM, periodic=PER)
    p, oid = oracle_parts(pos, vel, w), ids.copy()
    m = port.push(g, p, W.ef, dt, -O.QE, O.ME, ids=oid)
    gq, gi = by_id(e.getPartRef(), e.getPartRef()["id"])
    op, oi = by_id(p[:m], oid[:m])
    assert np.array_equal(gi, oi)
    d = np.abs(gq["pos"] - op["pos"])
    d[:, :2] = np.minimum(d[:, :2], np.abs(d[:, :2] - XM[:2]))  # a particle on the seam may lie at either end
    assert np.all(d <= 1e-5 * 1e-3)
    assert np.all(np.abs(gq["vel"] - op["vel"]) <= 1e-5 * np.abs(op["vel"]) + 1e-3)
    den = port.number_density(g, op)
    assert np.max(np.abs(e.den - den)) <= 1e-6 * np.max(den)
    W.close()
