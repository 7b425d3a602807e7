"""AC1D of photon lists over the walk's and the histograms' edges, against the
oracle: frames of 0, 1, 2 and 3 photons, batches on both sides of the planner's
own launch, shapes with and without room for the fixed-point histogram, counts,
bright counts past its range and values that are no counts.  Whole numbers match
exactly, the device route's uint64 histogram too; double sums within 1e-12 (their rounding, see test_gpu_ac1d_route)."""
import numpy as np
import pytest

from helpers import random_frames, small_detector

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("route", [0, 1])
@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("frames,size,values", [
    (1, 5, "counts"), (7, 40, "counts"), (40, 2048, "counts"), (40, 2048, "bright"), (40, 300, "floats"),
    (9, 7000, "counts"), (9, 8000, "counts"), (1024, 256, "counts"), (1025, 256, "floats"),
])
def test_ac1d_batches(ctx, oracle_lib, rng, frames, size, values, interp, route):
    import torch
    from incohautocorrelate_b200 import capi
    o = oracle_lib
    _, km, mq = small_detector(60, 64, 6e-4)
    sizes = ([0, 1, 2, 3, 64, 65, 200, 33] * (frames // 8 + 1))[:frames] if frames > 1 else [77]
    if frames > 100:
        sizes = [n // 8 for n in sizes]
    ph, off = random_frames(km, sizes, rng)
    if values == "bright":
        ph[:, 3] *= rng.integers(1, 4000, len(ph)).astype(np.float32)
    elif values == "floats":
        ph[:, 3] *= rng.uniform(1e-4, 3.0, len(ph)).astype(np.float32)
    sh = capi.ac1d_shape(mq, size)
    want = np.zeros(size, np.float64)
    o.lib().iaco_ac1d_uw_frames(o.p(np.ascontiguousarray(ph)), o.p(np.ascontiguousarray(off, np.uint64)), frames,
                                60 * 64, sh.max_q, sh.dq_per_step, size, interp, route, o.p(want))
    acc = torch.zeros(capi.ac1d_uw_words(sh), dtype=torch.int64, device="cuda")
    out = torch.zeros(size, dtype=torch.float64, device="cuda")
    ctx.ac1d_uw_batch(_dev(ph), _dev(off.astype(np.int64)), frames, 60 * 64, sh, interp, acc, route=route)
    ctx.ac1d_uw_finish(acc, sh, out)
    assert ctx.check() == 0
    got = out.cpu().numpy()
    if route == 1:  # the uint64 histogram; the oracle's doubles divide each frame's by 100 on its own
        vs = capi.ac1d_vecsize(sh.max_q, sh.dq_per_step)
        hist = np.zeros(vs, np.uint64)
        for f in range(frames):
            hl = np.ascontiguousarray(ph[off[f]:off[f + 1]])
            o.lib().iaco_ac1d_sparse_frame(o.p(hl), len(hl), sh.max_q, sh.dq_per_step, interp, 100.0, o.p(hist))
        np.testing.assert_array_equal(acc.cpu().numpy().view(np.uint64)[:vs], hist)
    elif interp == 0 and values != "floats":
        np.testing.assert_array_equal(got, want)
    else:
        np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)
