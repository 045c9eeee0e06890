"""The dot products of the persistent CG kernels, emulated exactly in FP32 on the CPU: FP32 over the 16 nodes that a
thread adds first, pairs of FP32 (48 bits) over everything above, scaled by a power of two.  Against FP64 they are no
further off than sums in FP32 over a thread and a warp of 1216 CTAs and FP64 above, and sums beyond FP32's range stay
finite.  Nor are those of the launch-per-pass kernels, whose threads sum more nodes in fewer CTAs."""
import numpy as np
import pytest

f32 = np.float32


def serial(x):
    """FP32 sums over the first axis, term by term."""
    s = np.zeros(x.shape[1:], f32)
    for t in x:
        s = (s + t).astype(f32)
    return s


def two_sum(a, b):
    s = (a + b).astype(f32)
    bb = (s - a).astype(f32)
    return s, ((a - (s - bb).astype(f32)).astype(f32) + (b - bb).astype(f32)).astype(f32)


def gather(h, l, h2, l2):  # ff_gather
    s, e = two_sum(h, h2)
    return s, (l + (l2 + e).astype(f32)).astype(f32)


def fold(h, l):
    """Pairs folded in halves over the last axis (the shuffles of a warp)."""
    while h.shape[-1] > 1:
        m = h.shape[-1] // 2
        h, l = gather(h[..., :m], l[..., :m], h[..., m:], l[..., m:])
    return two_sum(h[..., 0], l[..., 0])


def pad(x, m):
    return np.concatenate([x, np.zeros(-len(x) % m, f32)])


def launches(p, ctas=1216):
    """k_pcg_k2: a thread's groups of four in turn, a warp's tree, FP64."""
    threads = 256 * min(ctas, max(1, -(-(len(p) // 4) // 256)))
    s = serial(pad(p, 4 * threads).reshape(-1, threads, 4).transpose(0, 2, 1).reshape(-1, threads)).reshape(-1, 32)
    while s.shape[1] > 1:
        m = s.shape[1] // 2
        s = (s[:, :m] + s[:, m:]).astype(f32)
    return s.astype(np.float64).sum()


def launches_in_one_wave(p, ctas):
    """k_lpcg_k2 (456 CTAs), k_pcg_k2 (760): a thread's groups of four and its warp as pairs, FP64."""
    threads = 256 * min(ctas, max(1, -(-(len(p) // 4) // 256)))
    g = serial(pad(p, 4 * threads).reshape(-1, threads, 4).transpose(2, 0, 1))
    h, l = np.zeros(threads, f32), np.zeros(threads, f32)
    for t in g:
        h, e = two_sum(h, t)
        l = (l + e).astype(f32)
    h, l = h.reshape(-1, 32), l.reshape(-1, 32)
    while h.shape[1] > 1:
        m = h.shape[1] // 2
        h, l = gather(h[:, :m], l[:, :m], h[:, m:], l[:, m:])
    return h.astype(np.float64).sum() + l.astype(np.float64).sum()


def persistent(p, sms=152, threads=512):
    """k_pcg_grid: a thread's groups of four in turn in FP32, 16 nodes at a time; those, its warp, the warps of its CTA
    and the CTAs as pairs."""
    chunk = -(-(-(-len(p) // sms)) // 32) * 32
    groups = -(-chunk // (16 * threads)) * 4
    x = np.zeros((sms, groups * 4 * threads), f32)
    x[:, :chunk] = pad(p, sms * chunk).reshape(sms, chunk)
    x = x.reshape(sms, groups // 4, 4, threads, 4).transpose(2, 4, 1, 0, 3)  # group of 16, node; 16 nodes, CTA, thread
    g = serial(x.reshape(16, groups // 4, sms, threads))
    h, l = np.zeros_like(g[0]), np.zeros_like(g[0])
    for t in g:
        h, e = two_sum(h, t)
        l = (l + e).astype(f32)
    k = f32(2.0 ** -np.floor(np.log2(p.astype(np.float64).sum())))  # sum_scales
    h, l = fold(h.reshape(sms, -1, 32), l.reshape(sms, -1, 32))
    h, l = (h * k).astype(f32), (l * k).astype(f32)
    fill = 32 - h.shape[1]
    h, l = fold(np.pad(h, ((0, 0), (0, fill))), np.pad(l, ((0, 0), (0, fill))))
    th, tl = np.zeros(32, f32), np.zeros(32, f32)
    for b in range(0, sms, 32):
        m = min(32, sms - b)
        th[:m], tl[:m] = gather(th[:m], tl[:m], h[b:b + m], l[b:b + m])
    h, l = fold(th, tl)
    return (float(h) + float(l)) / float(k)


@pytest.mark.parametrize("n", [9261, 40_000, 98_000, 274_625, 1_000_000, 2_146_689])
def test_no_further_from_fp64_than_the_launches(n):
    rng = np.random.default_rng(n)
    a, b = [], []
    for _ in range(6):
        r = (rng.normal(size=n) * np.exp(rng.normal(size=n))).astype(f32)
        p = (r * r).astype(f32)
        exact = p.astype(np.float64).sum()
        a.append(launches(p) / exact - 1)
        b.append(persistent(p) / exact - 1)
    assert np.sqrt(np.mean(np.square(b))) <= np.sqrt(np.mean(np.square(a)))


@pytest.mark.parametrize("ctas", [456, 760])
@pytest.mark.parametrize("n", [1_000_003, 2_146_689, 8_000_000])
def test_one_wave_of_launches_is_no_further_from_fp64(n, ctas):
    rng = np.random.default_rng(n)
    a, b = [], []
    for _ in range(3):
        r = (rng.normal(size=n) * np.exp(rng.normal(size=n))).astype(f32)
        p = (r * r).astype(f32)
        exact = p.astype(np.float64).sum()
        a.append(launches(p) / exact - 1)
        b.append(launches_in_one_wave(p, ctas) / exact - 1)
    assert np.sqrt(np.mean(np.square(b))) <= np.sqrt(np.mean(np.square(a)))


def test_sums_beyond_the_range_of_fp32():
    r = np.full(100_000, 4e17, f32)
    p = (r * r).astype(f32)
    assert p.astype(np.float64).sum() > 3.4e38
    assert abs(persistent(p) / p.astype(np.float64).sum() - 1) < 1e-7
