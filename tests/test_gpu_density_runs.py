"""pic_number_density_noalloc sums runs of particles of one cell before they reach the accumulator: counts
around the runs' and turns' edges, in cell order, scattered, in one cell, along x and with particles that
are to be skipped, against a numpy restatement.  The sums are integers: every bit has to agree."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NN, PER, SCALE = (14, 9, 11), (1, 0, 1), 2.0 ** 20


def expected(cell, off, w, live):
    f = np.float32
    acc = np.zeros(int(np.prod(NN)), np.uint64)
    c, o, s = cell[live], off[live], w[live] * f(SCALE)
    base = (c[:, 2] * NN[1] + c[:, 1]) * NN[0] + c[:, 0]
    for m in range(8):
        wx, wy, wz = [o[:, d] if (m >> d) & 1 else f(1) - o[:, d] for d in range(3)]
        v = np.rint(s * wx * wy * wz).astype(np.uint64)
        np.add.at(acc, base + (m & 1) + NN[0] * ((m >> 1) & 1) + NN[0] * NN[1] * (m >> 2), v)
    a = acc.reshape(NN[::-1]).copy()
    inv_vol = np.full(a.shape, 1.0 / (1.0 / (NN[0] - 1) * (1.0 / (NN[1] - 1)) * (1.0 / (NN[2] - 1))))
    for d in range(3):
        first, last = [slice(None)] * 3, [slice(None)] * 3
        first[2 - d], last[2 - d] = 0, NN[d] - 1
        if PER[d]:
            a[tuple(first)] += a[tuple(last)]
            a[tuple(last)] = a[tuple(first)]
        else:
            inv_vol[tuple(first)] *= 2
            inv_vol[tuple(last)] *= 2
    return (a.astype(np.float64) * ((1.0 / SCALE) * inv_vol)).astype(np.float32)


@pytest.mark.parametrize("order", ["cells", "random", "one_cell", "along_x", "holes"])
@pytest.mark.parametrize("n", [0, 1, 33, 1000, 155_647, 155_649, 622_600, 5_000_000])
def test_density_equals_integer_sums(pic, n, order):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + len(order))
    cell = np.stack([rng.integers(0, k - 1, n) for k in NN], 1)
    if order == "one_cell":
        cell[:] = (5, 3, 2)
    elif order == "along_x":
        cell = np.stack([np.arange(n) // 3 % (NN[0] - 1), np.full(n, 2), np.full(n, 4)], 1)
    elif order != "random":
        cell = cell[np.lexsort((cell[:, 0], cell[:, 1], cell[:, 2]))]
    off = rng.random((n, 3), dtype=np.float32)
    w = (20 * np.exp(0.5 * rng.standard_normal(n))).astype(np.float32)
    packed = (cell[:, 0] | cell[:, 1] << 9 | cell[:, 2] << 18).astype(np.int32)
    live = np.ones(n, bool)
    if order == "holes":  # removed particles and cells outside the grid, within runs and at their ends
        gone, outside = rng.random(n) < 0.3, rng.random(n) < 0.1
        packed[outside] = np.int32(NN[0] - 1)
        packed[gone] = -1
        live = ~(gone | outside)
    p4 = np.concatenate([off, packed.view(np.float32)[:, None]], 1)
    v4 = np.concatenate([rng.random((n, 3), dtype=np.float32), w[:, None]], 1)
    p4, v4 = torch.from_numpy(p4).cuda(), torch.from_numpy(v4).cuda()
    out = torch.full((int(np.prod(NN)),), -1.0, device="cuda")
    x0, xm, per = np.zeros(3), np.ones(3), np.array(PER, np.int32)
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    rc = pic.library().pic_number_density_noalloc(
        *NN, x0.ctypes.data_as(C.c_void_p), xm.ctypes.data_as(C.c_void_p), per.ctypes.data_as(C.c_void_p), ptr(p4),
        ptr(v4), n, SCALE, ptr(out), None)
    assert rc == pic.PIC_OK
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().reshape(NN[::-1]), expected(cell, off, w, live))
