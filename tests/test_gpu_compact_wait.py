"""Uploads whose compaction waits in vain: the call reports it, and exactly the particles inside the box are
there, as after an upload whose wait ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n,out", [(3, 2), (5_000, 7), (400_000, 2), (5_000, 0)])
def test_wait_that_runs_out_is_reported_and_particles_stay_whole(pic, n, out, pinned):
    torch = pytest.importorskip("torch")
    W = pic.World(17, 17, 17, (0.0, 0.0, 0.0), (0.016, 0.016, 0.016))
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 0.016, (n, 3)) * 0.999999
    if out:
        pos[::out] = 0.02  # outside: dropped by the rewinding upload
    vel, w = rng.normal(size=(n, 3)) * 1e5, rng.uniform(1.0, 2.0, n)
    ids = rng.permutation(n).astype(np.uint64)
    arrays = [pos, vel, w]
    if pinned:
        arrays = [torch.from_numpy(a).pin_memory().numpy() for a in arrays]
    whole = pic.Species("a", pic.ME, -pic.QE, W, 1.5, capacity=n)
    whole.addParticles(*arrays, ids=ids, rewind=True)
    short = pic.Species("b", pic.ME, -pic.QE, W, 1.5, capacity=n)
    assert W._L.pic_debug_set_wait_polls(W._h, 0) == pic.PIC_OK
    try:
        if out:
            with pytest.raises(pic.PicError) as ei:
                short.addParticles(*arrays, ids=ids, rewind=True)
            assert ei.value.code == pic.PIC_ERR_DEVICE and "bounded wait" in str(ei.value)
        else:  # nothing to remove, nothing to wait for
            short.addParticles(*arrays, ids=ids, rewind=True)
    finally:
        assert W._L.pic_debug_set_wait_polls(W._h, -1) == pic.PIC_OK
    a, b = whole.getPartRef(), short.getPartRef()
    a, b = a[np.argsort(a["id"])], b[np.argsort(b["id"])]
    assert len(a) == (n - len(pos[::out]) if out else n)
    for f in ("id", "pos", "vel", "w"):
        assert np.array_equal(a[f], b[f])
    W.close()
