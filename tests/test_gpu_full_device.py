"""A device whose memory is used up: node fields, densities and gas properties go through the little staging that a
world always has, and the learned preconditioner does without its dense matrix."""
import contextlib
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def used_up(free):
    """All device memory held but for blocks below `free` bytes and one block of `free`."""
    pytest.importorskip("torch")  # has the CUDA runtime in the process
    rt = C.CDLL("libcudart.so.13")
    spare = C.c_void_p()
    assert rt.cudaMalloc(C.byref(spare), C.c_size_t(free)) == 0
    held, size = [], 1 << 34
    while size >= free:
        p = C.c_void_p()
        if rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
            held.append(p)
        else:
            size >>= 1
    rt.cudaGetLastError()
    rt.cudaFree(spare)
    try:
        yield
    finally:
        for p in held:
            rt.cudaFree(p)


def make(pic, nn):
    W = pic.World(*nn, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    s = pic.Species("O", 16 * pic.AMU, 0.0, W, 1e3, capacity=50_000)
    s.loadUniform((0, 0, 0), (1, 1, 1), 50_000, 300.0, 1e3, 0.0, seed=3)
    s.advance(1e-9, deposit=True)
    W.computeChargeDensity()
    s.updateAverages()
    s.sampleMoments()
    return W, s


def write(W):
    rng = np.random.default_rng(2)
    W.phi, W.rho, W.ef = rng.normal(size=W.nv), rng.normal(size=W.nv), rng.normal(size=(W.nv, 3))


def read(W, s):
    return [W.phi, W.rho, W.ef, s.den, s.den_avg, *s.computeGasProperties()]


def test_fields_without_device_memory(pic):
    small, ss = make(pic, (9, 9, 9))  # every kernel of the test has run once: their code is loaded
    write(small)
    read(small, ss)
    W, s = make(pic, (97, 99, 101))  # 7.8 MB of potential, no field of it moved yet
    with used_up(1 << 20):
        write(W)
        short = read(W, s)
    for a, b in zip(short, read(W, s)):
        assert np.array_equal(a, b)
    write(W)
    for a, b in zip(short, read(W, s)):
        assert np.array_equal(a, b)
    W.close()
    small.close()


def test_learned_preconditioner_with_little_device_memory(pic):
    """Room for the levels but not for the dense matrix of the coarse ones (16 MB): each is applied by itself, within
    the bound of the tests of the levels."""
    import learned_ref as LR
    from test_gpu_learned import distinct, free_mask, unpack

    nn, per, xm = (48, 52, 52), (0, 0, 0), (0.047, 0.051, 0.051)  # levels of 24 x 26 x 26, 12 x 13 x 13, ..
    r = np.random.default_rng(4).normal(size=int(np.prod(nn)))

    def world():
        W = pic.World(*nn, (0.0, 0.0, 0.0), xm)
        W.set_boundaries(per, (1,) * 6, (0.0,) * 6)
        W.rho = r * 1e-7
        return W

    def learned(W):
        lp, S = pic.LearnedPreconditioner(W), pic.PotentialSolver(W, 2000, 1e-8, pic.SOLVER_LEARNED)
        z = lp.apply(r)
        assert S.solve(raise_on_fail=True)
        return lp, z, W.phi

    warm = world()
    lp, full, phi = learned(warm)  # the kernels' code is loaded
    w = lp.weights()
    assert lp.levels()[0][2] == (12, 13, 13)
    little = world()
    phi0 = little.phi
    assert pic.PotentialSolver(little, 5000, 1e-6, pic.SOLVER_PCG).solve()  # what every solver allocates is there
    little.phi = phi0
    with used_up(1 << 22):
        _, z, phi1 = learned(little)
    g = dict(nn=nn, per=per, xm=xm)
    ref = LR.apply(distinct(r, g), free_mask(g), unpack(w), (False,) * 3, lp.levels()[1])
    for v in (z, full):
        assert np.max(np.abs(distinct(v, g) - ref)) <= 2e-5 * np.max(np.abs(ref))
    # two residuals of 1e-8 through the operator's condition number, 4 N^2 / pi^2 = 1.1e3 for N = 52
    assert np.max(np.abs(phi1 - phi)) <= 2e-8 * 1.1e3 * np.max(np.abs(phi))
    warm.close()
    little.close()
