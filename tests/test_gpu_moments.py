"""Velocity moments and gas properties: the sampling kernel sums runs of consecutive particles of a
cell in registers, so it is compared with FP64 sums for particles in cell order, in random order and
alternating between two cells, at counts around a run and a block, on odd grids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fp64_moments(nn, x0, xm, pos, vel, w):
    """n, n v, n v^2 (7 x nodes) with the CIC weights in FP64, and the sums of |terms| (Species.cpp:767-776)."""
    nn = np.asarray(nn)
    lc = (pos - x0) / ((np.asarray(xm) - x0) / (nn - 1))
    c = np.minimum(lc.astype(int), nn - 2)
    f = lc - c
    val = np.stack([w, *(w * vel.T), *(w * vel.T ** 2)])
    m, a = np.zeros((7, np.prod(nn))), np.zeros((7, np.prod(nn)))
    for k in range(8):
        b = [(k >> d) & 1 for d in range(3)]
        wt = np.prod([f[:, d] if b[d] else 1 - f[:, d] for d in range(3)], axis=0)
        node = ((c[:, 2] + b[2]) * nn[1] + c[:, 1] + b[1]) * nn[0] + c[:, 0] + b[0]
        for q in range(7):
            np.add.at(m[q], node, wt * val[q])
            np.add.at(a[q], node, np.abs(wt * val[q]))
    return m, a


@pytest.mark.parametrize("order", ["cells", "random", "alternating"])
@pytest.mark.parametrize("n", [1, 15, 17, 129, 50_001])
def test_moments_of_runs_match_fp64(pic, order, n):
    nn, x0, xm = (6, 9, 5), np.zeros(3), np.array([0.5, 0.8, 0.4])
    rng = np.random.default_rng(n)
    pos = (rng.uniform(0, 1, (n, 3)).astype(np.float32) * 0.999).astype(np.float64) * xm
    if order == "alternating":  # two cells in turn: every particle ends its predecessor's run
        pos = (rng.uniform(0.05, 0.95, (n, 3)) + np.where(np.arange(n)[:, None] % 2, [4, 7, 3], [0, 1, 0])) * 0.1
    if order == "cells":
        c = np.floor(pos / 0.1).astype(int)
        pos = pos[np.lexsort((c[:, 0], c[:, 1], c[:, 2]))]
    vel = rng.normal(size=(n, 3)).astype(np.float32).astype(np.float64) * 512.0 + 256.0
    w = rng.uniform(0.5, 2.0, n).astype(np.float32).astype(np.float64)
    W = pic.World(*nn, x0, xm)
    sp = pic.Species("O", pic.AMU, 0.0, W, 1.0, capacity=n + 8)
    sp.addParticles(pos, vel, w, rewind=False)
    sp.sampleMoments()
    gv, gT = sp.computeGasProperties()
    m, a = fp64_moments(nn, x0, xm, pos, vel, w)
    # a node's FP32 sum of K terms: at most (K + 8) roundings of 2^-24 of the sum of |terms| (the terms'
    # own five products included), and in-cell offsets within 2^-23 of a cell, which move a corner weight
    # by up to 3 * 2^-23 absolutely: small against the node's weight where that exceeds 1 % of a particle
    live = m[0] > 0.02
    eps = (min(n, 4000) + 8) * 2.0**-24 + 3 * 2.0**-23 * 8 * n / np.maximum(m[0], 0.02)
    u = m[1:4] / np.where(live, m[0], 1)
    du = 2 * eps * (a[1:4] / np.where(live, m[0], 1) + np.abs(u))
    assert np.all(np.abs(gv.T - u)[:, live] <= du[:, live])
    T = pic.AMU / (2 * pic.KB) * (m[4:7] / np.where(live, m[0], 1) - u**2).sum(0)
    dT = pic.AMU / (2 * pic.KB) * (2 * eps * a[4:7] / np.where(live, m[0], 1) * 2 + 2 * np.abs(u) * du + du**2).sum(0)
    assert np.all(np.abs(gT - T)[live] <= dT[live])
    W.close()
