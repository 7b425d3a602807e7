"""Dense C(q) and AC1D tiles whose values stay below 2^23 (their own kernels'
path) next to tiles that leave it, bit for bit against the oracle: values at
the limit, negative intensities, masked pixels whose k is far outside the mesh,
MaxQ cuts, ragged tiles, Multiplicators that are no integers or no floats."""
import numpy as np
import pytest

from helpers import small_detector, to_capi_shape

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _cases(rng, npix, km):
    """(name, I, kmap, Multiplicator)"""
    I = rng.uniform(0.05, 1.5, npix).astype(np.float32)
    I[rng.random(npix) < 0.1] = 0
    edge = I.copy()
    top = float(edge.max())
    limit = 2.0 ** 23 / top ** 2  # the tiles of the brightest pixel end just past the limit, others below
    far = km.copy().reshape(-1, 3)
    far[I == 0] = np.float32(1e18)
    negative = I.copy()
    negative[3::97] *= -1
    dim = (I * np.float32(1e-18)).astype(np.float32)  # products around the 1e-37 cut
    yield "limit", edge, km, float(np.floor(limit))
    yield "past", edge, km, float(np.ceil(limit) + 1)
    yield "fraction", I, km, 100000.5
    yield "no float", I, km, 16777217.0
    yield "far masked", I, far.reshape(-1), 123457.0
    yield "negative", negative, km, 100000.0
    yield "dim", dim, km, 2.0 ** 29 - 1
    yield "huge", dim, km, 1e38
    yield "all masked", np.zeros(npix, np.float32), km, 1000.0


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("ny,nx,cut", [(16, 16, 1.0), (17, 31, 0.6), (40, 33, 1.0)])
def test_cq_small_values(ctx, oracle_lib, rng, interp, ny, nx, cut):
    o = oracle_lib
    _, km, mq = small_detector(ny, nx, 6e-4)
    npix = ny * nx
    s = o.small_cq_mesh_shape(mq, 41)
    s.max_q = np.float32(cut) * s.max_q
    for name, I, k, mult in _cases(rng, npix, km):
        want = np.zeros(s.size_ab * s.size_ab * s.size_c, np.uint64)
        o.lib().iaco_cq_small(o.p(I), o.p(k), npix, s, interp, mult, 0, npix, o.p(want))
        for fast in (0, nx):
            out = _dev(np.zeros(want.size, np.int64))
            ctx.cq_small(_dev(I), _dev(k), npix, to_capi_shape(s), interp, mult, out, fast_size=fast)
            np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want, err_msg=f"{name} {fast}")


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("ny,nx,size,cut", [(16, 16, 3, 1.0), (17, 31, 300, 0.6), (40, 33, 1000, 1.0)])
def test_ac1d_small_values(ctx, oracle_lib, rng, interp, ny, nx, size, cut):
    from incohautocorrelate_b200 import capi
    o = oracle_lib
    _, km, mq = small_detector(ny, nx, 6e-4)
    npix = ny * nx
    so, sh = o.ac1d_shape(mq, size), capi.ac1d_shape(mq, size)
    max_q = np.float32(cut * sh.max_q)
    for wrap in (1.0, 0.7):  # 0.7: bins past the histogram wrap around it
        for s in (so, sh):
            s.max_q = max_q
            s.dq_per_step = np.float32(max_q / (size - 1.5) * wrap)
        for name, I, k, mult in _cases(rng, npix, km):
            want = np.zeros(sh.size, np.uint64)
            o.lib().iaco_ac1d_cq(o.p(I), o.p(k), npix, so, interp, mult, 0, npix, o.p(want))
            out = _dev(np.zeros(want.size, np.int64))
            ctx.ac1d_cq(_dev(I), _dev(k), npix, sh, interp, mult, out)
            np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want, err_msg=f"{name} {wrap}")


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("edge", [25, 45, 61, 81, 121])
def test_cq_small_window_sizes(ctx, oracle_lib, rng, interp, edge):
    """Meshes whose tile windows fill a part of the shared-memory window, just
    fit it, or exceed it in some or all tile pairs."""
    o = oracle_lib
    ny, nx = 37, 44
    _, km, mq = small_detector(ny, nx, 6e-4)
    I = rng.uniform(0.05, 1.5, ny * nx).astype(np.float32)
    s = o.small_cq_mesh_shape(mq, edge)
    want = np.zeros(s.size_ab * s.size_ab * s.size_c, np.uint64)
    o.lib().iaco_cq_small(o.p(I), o.p(km), ny * nx, s, interp, 123457.0, 0, ny * nx, o.p(want))
    for fast in (0, nx):
        out = _dev(np.zeros(want.size, np.int64))
        ctx.cq_small(_dev(I), _dev(km), ny * nx, to_capi_shape(s), interp, 123457.0, out, fast_size=fast)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want, err_msg=str(fast))


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("case", ["far pixels", "window product past 2^31", "coordinates past 2^22"])
def test_cq_window_past_the_integers(ctx, oracle_lib, rng, interp, case):
    """Tile pairs whose q range the window's integers cannot hold: pixels whose k is
    finite but far off, a window of 1 480 voxels on each axis, and a small window at
    voxel 2^23.  What lies outside the mesh is skipped, the rest is the oracle's."""
    o = oracle_lib
    npix = 3 * 256 + 17
    s = o.small_cq_mesh_shape(np.array([1.0, 0.9, 0.4], np.float32), 41)
    k = rng.uniform(0.0, 0.01, (npix, 3)).astype(np.float32)
    s.voxel_per_dq, s.max_q = 1500, np.float32(4.0)
    if case == "far pixels":
        k[5::64] = np.float32(1e18)
        k[37::64] = np.float32(-1e18)
    elif case == "window product past 2^31":
        s.voxel_per_dq = 740
        k = rng.uniform(0.0, 1.0, (npix, 3)).astype(np.float32)
        k[::5] = k[0] + rng.uniform(0.0, 0.01, (len(k[::5]), 3)).astype(np.float32)
    else:
        s.voxel_per_dq = 1 << 23
        k = rng.uniform(0.0, 1e-6, (npix, 3)).astype(np.float32)
        k[256:512, 0] += np.float32(1.0)
    I = rng.uniform(0.05, 1.5, npix).astype(np.float32)
    want = np.zeros(s.size_ab * s.size_ab * s.size_c, np.uint64)
    k = np.ascontiguousarray(k.reshape(-1))
    o.lib().iaco_cq_small(o.p(I), o.p(k), npix, s, interp, 1000.0, 0, npix, o.p(want))
    assert want.any()
    out = _dev(np.zeros(want.size, np.int64))
    ctx.cq_small(_dev(I), _dev(k), npix, to_capi_shape(s), interp, 1000.0, out)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)
    ctx.check()


@pytest.mark.parametrize("interp", [0, 1])
def test_cq_maxq_that_bounds_nothing(ctx, oracle_lib, rng, interp):
    """A MaxQ that is no number or infinite: every pair counts, as |q| > MaxQ is false."""
    o = oracle_lib
    _, km, mq = small_detector(17, 31, 6e-4)
    I = rng.uniform(0.05, 1.5, 17 * 31).astype(np.float32)
    s = o.small_cq_mesh_shape(mq, 41)
    for s.max_q in (np.nan, np.inf):
        want = np.zeros(s.size_ab * s.size_ab * s.size_c, np.uint64)
        o.lib().iaco_cq_small(o.p(I), o.p(km), I.size, s, interp, 123457.0, 0, I.size, o.p(want))
        assert want.any()
        out = _dev(np.zeros(want.size, np.int64))
        ctx.cq_small(_dev(I), _dev(km), I.size, to_capi_shape(s), interp, 123457.0, out, fast_size=31)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)
    ctx.check()


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("lit", [0.004, 0.05, 0.5, 1.0])
@pytest.mark.parametrize("sign", ["positive", "some negative", "bright"])
def test_maps_of_few_lit_pixels(ctx, oracle_lib, rng, interp, lit, sign):
    """Tiles of which none, one, an odd number, most or all pixels are lit, in both
    dense kernels: values of every kind, the masked pixels' k far outside."""
    from incohautocorrelate_b200 import capi
    o = oracle_lib
    ny, nx = 37, 44
    _, km, mq = small_detector(ny, nx, 6e-4)
    I = rng.uniform(0.05, 1.5, ny * nx).astype(np.float32)
    I[rng.random(I.size) >= lit] = 0
    I[-1] = 1.0
    if sign == "some negative":
        I[::3] *= -1
    elif sign == "bright":
        I[::5] *= 3000
    k = km.copy().reshape(-1, 3)
    k[I == 0] = np.float32(1e18)
    k = np.ascontiguousarray(k.reshape(-1))
    s = o.small_cq_mesh_shape(mq, 41)
    want = np.zeros(s.size_ab * s.size_ab * s.size_c, np.uint64)
    o.lib().iaco_cq_small(o.p(I), o.p(k), I.size, s, interp, 123457.0, 0, I.size, o.p(want))
    for fast in (0, nx):
        out = _dev(np.zeros(want.size, np.int64))
        ctx.cq_small(_dev(I), _dev(k), I.size, to_capi_shape(s), interp, 123457.0, out, fast_size=fast)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want, err_msg=str(fast))
    for mult in (123457.0, 100000.5):
        so, sh = o.ac1d_shape(mq, 300), capi.ac1d_shape(mq, 300)
        want = np.zeros(sh.size, np.uint64)
        o.lib().iaco_ac1d_cq(o.p(I), o.p(k), I.size, so, interp, mult, 0, I.size, o.p(want))
        out = _dev(np.zeros(want.size, np.int64))
        ctx.ac1d_cq(_dev(I), _dev(k), I.size, sh, interp, mult, out)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want, err_msg=str(mult))
