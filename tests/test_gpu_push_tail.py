"""The push where a CTA goes from a full chunk to the last, partial one: the full chunk is still being
stored from the shared memory that the tail is read into.  The smallest launch shape gives every CTA two full
chunks and the first one the tail too; all particles are compared with the FP64 oracle by id, with the
tolerances of the parity tests."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import by_id, oracle_parts, smooth_field

pytestmark = pytest.mark.gpu

NN, PER = (37, 23, 45), (1, 1, 0)
XM = (0.036, 0.022, 0.044)
CHUNK, CTAS_PER_SM = 512, 2  # particles of a chunk, the kernel's CTAs an SM of the smallest shape


@pytest.mark.parametrize("deposit", [True, False])
@pytest.mark.parametrize("tail", [1, 300, 511])
def test_tail_after_full_chunks_matches_the_oracle(pic, port, tail, deposit):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 2 * CTAS_PER_SM * sms * CHUNK + tail
    rng = np.random.default_rng(tail)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * XM * (1, 1, 0.98) + (0, 0, 0.01 * XM[2])
    c = np.floor(pos / 1e-3).astype(int)
    pos = pos[np.lexsort((c[:, 0], c[:, 1], c[:, 2]))]
    vel = rng.normal(0.0, 4e5, (n, 3))
    w = rng.lognormal(0.0, 0.5, n) * 64.0
    dt = 8e-10
    W = pic.World(*NN, (0.0, 0.0, 0.0), XM)
    W.set_boundaries(PER, (1,) * 6, (0.0,) * 6)
    W.ef = smooth_field(int(np.prod(NN)), NN, None, 50.0, 3)
    W.set_launch_shapes(1)
    e = pic.Species("e-", pic.ME, -pic.QE, W, 64.0, capacity=n + 16)
    ids = np.arange(n, dtype=np.uint64)
    e.addParticles(pos, vel, w, ids=ids, rewind=False)
    e.advance(dt, deposit=deposit)
    g = port.grid(NN, (0.0, 0.0, 0.0), XM, periodic=PER)
    p, oid = oracle_parts(pos, vel, w), ids.copy()
    m = port.push(g, p, W.ef, dt, -O.QE, O.ME, ids=oid)
    gp = e.getPartRef()
    gq, gi = by_id(gp, gp["id"])
    op, oi = by_id(p[:m], oid[:m])
    assert np.array_equal(gi, oi)
    d = np.abs(gq["pos"] - op["pos"])
    d[:, :2] = np.minimum(d[:, :2], np.abs(d[:, :2] - XM[:2]))  # a particle on the seam may lie at either end
    assert np.all(d <= 1e-5 * 1e-3)
    assert np.all(np.abs(gq["vel"] - op["vel"]) <= 1e-5 * np.abs(op["vel"]) + 1e-3)
    if deposit:
        W.computeChargeDensity()
        den = port.number_density(g, op)
        assert np.max(np.abs(e.den - den)) <= 1e-6 * np.max(den)
    W.close()
