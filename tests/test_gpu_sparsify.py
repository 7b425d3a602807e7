"""iac_sparsify_frames (CreateSparseHitList, IAC/Detector.cpp:926-977) where its
tiles and ranks can go wrong, bit for bit against the same selection in numpy:
detectors around the tile of 4 096 pixels, rows that allow 16-byte loads and
rows that do not, no hits and only hits, a list that does not fit its capacity,
and a context whose scratch has no room for the bits between the two passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def want_lists(x, mask, km, thr, step, photonize):
    v = x if mask is None else x * mask.astype(np.float32)[None, :]
    hit = (v >= np.float32(thr)) & (v > 0)
    f, p = np.nonzero(hit)
    val = v[f, p]
    if photonize:
        val = np.ceil((val - np.float32(thr)) / np.float32(step)).astype(np.float32)
    out = np.concatenate([km.reshape(-1, 3)[p], val[:, None]], 1).astype(np.float32)
    return out, np.concatenate([[0], np.cumsum(hit.sum(1))]).astype(np.int64)


def run(ctx, x, mask, km, thr, step, photonize, cap, total=True):
    import torch
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    nf, npix = x.shape
    out = torch.full((max(cap, 1), 4), -7.0, dtype=torch.float32, device="cuda")
    off = torch.zeros(nf + 1, dtype=torch.int64, device="cuda")
    n = ctx.sparsify_frames(dev(x), None if mask is None else dev(mask), dev(km), npix, nf, thr, step, photonize, out,
                            cap, off, want_total=total)
    return out.cpu().numpy(), off.cpu().numpy(), n


@pytest.mark.parametrize("npix", [1, 31, 4095, 4096, 4097, 4 * 1024 * 3, 9973])
@pytest.mark.parametrize("nframes", [1, 5])
@pytest.mark.parametrize("share", [0.0, 0.01, 1.0])
@pytest.mark.parametrize("masked,photonize", [(False, 1), (True, 1), (True, 0)])
def test_lists_match(ctx, rng, npix, nframes, share, masked, photonize):
    km = rng.normal(size=(npix, 3)).astype(np.float32)
    x = np.where(rng.random((nframes, npix)) < share, rng.gamma(2.0, 1.0, (nframes, npix)) + 0.5, -0.3).astype(np.float32)
    mask = (rng.random(npix) > 0.1).astype(np.int32) if masked else None
    want, off_w = want_lists(x, mask, km, 0.5, 0.73, photonize)
    got, off, n = run(ctx, x, mask, km, 0.5, 0.73, photonize, nframes * npix)
    assert n == len(want)
    np.testing.assert_array_equal(off, off_w)
    np.testing.assert_array_equal(got[:n], want)
    assert (got[n:] == -7.0).all()
    assert ctx.check() == 0


def test_many_tiles_and_frames(ctx, rng):
    """More counts than one round of the scan takes."""
    npix, nframes = 4100, 3000
    km = rng.normal(size=(npix, 3)).astype(np.float32)
    x = np.where(rng.random((nframes, npix)) < 0.002, 1.0, 0.0).astype(np.float32)
    want, off_w = want_lists(x, None, km, 0.0, 1.0, 1)
    got, off, n = run(ctx, x, None, km, 0.0, 1.0, 1, 60000)
    np.testing.assert_array_equal(off, off_w)
    np.testing.assert_array_equal(got[:n], want)


def test_capacity_is_never_passed(ctx, rng):
    from incohautocorrelate_b200 import capi
    npix, nframes, cap = 5000, 6, 777
    km = rng.normal(size=(npix, 3)).astype(np.float32)
    x = (rng.random((nframes, npix)) < 0.05).astype(np.float32)
    want, off_w = want_lists(x, None, km, 0.0, 1.0, 1)
    got, off, _ = run(ctx, x, None, km, 0.0, 1.0, 1, cap, total=False)
    np.testing.assert_array_equal(got, want[:cap])
    np.testing.assert_array_equal(off, np.minimum(off_w, cap))
    with pytest.raises(capi.IacError) as e:
        ctx.check()
    assert e.value.status == capi.IAC_ERR_NO_MEMORY and str(len(want) - cap) in str(e.value)


def test_without_room_for_the_bits(rng):
    """A scratch limit that holds the counts and offsets only: the frames are read
    twice, and the lists stay the same."""
    from incohautocorrelate_b200 import capi
    npix, nframes = 9000, 7
    km = rng.normal(size=(npix, 3)).astype(np.float32)
    x = np.where(rng.random((nframes, npix)) < 0.03, 2.3, 0.1).astype(np.float32)
    mask = (rng.random(npix) > 0.1).astype(np.int32)
    want, off_w = want_lists(x, mask, km, 0.5, 1.0, 1)
    c = capi.Context(0)
    try:
        c.set_scratch_limit(2048)
        got, off, n = run(c, x, mask, km, 0.5, 1.0, 1, nframes * npix)
        np.testing.assert_array_equal(off, off_w)
        np.testing.assert_array_equal(got[:n], want)
        assert c.check() == 0
    finally:
        c.close()
