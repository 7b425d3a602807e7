"""The pair kernel's walk and fast paths where they can go wrong, bit for bit
against the oracle's half mesh (integers): photon counts around the edges of the
32-lane units and of the step chunks, batches planned by the kernel itself (up
to 256 frames) and by the planner, every size of the shared-memory box with
sums past 32 bits, and batches that mix frames of the fast path with frames
that must not take it."""
import numpy as np
import pytest

from helpers import random_frames, small_detector, to_capi_shape

pytestmark = pytest.mark.gpu


def want_half(o, ph, off, rot, shape, dmap, i1, i2, mult=1000.0):
    half = np.zeros(o.half_words(shape.size_ab), np.uint64)
    oob = 0
    for f in range(len(off) - 1):
        hl = np.ascontiguousarray(ph[int(off[f]):int(off[f + 1])])
        if len(hl):
            P = o.sparse_params_array(shape, len(hl), dmap, i1, i2, mult)
            oob += o.lib().iaco_sparse_ac_halfmesh(o.p(hl), len(hl), o.p(P), o.p(np.ascontiguousarray(rot[f])), o.p(half))
    return half, oob


def gpu_half(ctx, ph, off, rot, shape, dmap, i1, i2, mult=1000.0):
    import torch
    from incohautocorrelate_b200 import capi
    half = torch.zeros(capi.half_mesh_words(shape.size_ab), dtype=torch.int64, device="cuda")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ctx.sparse_ac_batch(dev(ph), dev(off.astype(np.int64)), dev(rot.astype(np.float32)), len(off) - 1,
                        capi.sparse_params(to_capi_shape(shape), i1, i2, dmap, mult), half)
    return half, ctx.check()


def check(ctx, o, ph, off, rot, shape, dmap, i1, i2, mult=1000.0):
    want, o1 = want_half(o, ph, off, rot, shape, dmap, i1, i2, mult)
    got, o2 = gpu_half(ctx, ph, off, rot, shape, dmap, i1, i2, mult)
    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint64), want)
    assert o1 == o2


MODES = [(1, 0, 0), (0, 0, 0), (0, 0, 1), (1, 0, 1), (1, 1, 0), (1, 1, 1)]
EDGES = [0, 1, 2, 3, 4, 31, 32, 33, 63, 64, 65, 66, 67, 127, 128, 129, 130, 131, 193, 0, 257]


@pytest.mark.parametrize("dmap,i1,i2", MODES)
@pytest.mark.parametrize("pad", [0, 240], ids=["planned_by_the_kernel", "planner"])
@pytest.mark.parametrize("integer", [True, False])
def test_unit_and_chunk_edges(ctx, oracle_lib, rng, dmap, i1, i2, pad, integer):
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    shape = oracle_lib.big_mesh_shape(mq, 31)
    sizes = EDGES + [0, 1, 2] * (pad // 3)
    ph, off = random_frames(km, sizes, rng, integer=integer)
    check(ctx, oracle_lib, ph, off, W.haar_rotations(len(sizes), seed=3), shape, dmap, i1, i2)


@pytest.mark.parametrize("frames", [255, 256, 257])
def test_frame_counts_around_the_planner(ctx, oracle_lib, rng, frames):
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    shape = oracle_lib.big_mesh_shape(mq, 31)
    ph, off = random_frames(km, rng.integers(0, 40, frames), rng)
    check(ctx, oracle_lib, ph, off, W.haar_rotations(frames, seed=4), shape, 1, 0, 0)


@pytest.mark.parametrize("frames", [2, 3, 30, 300])
@pytest.mark.parametrize("values", ["counts", "counts to 128", "real", "past 32 bits"])
@pytest.mark.parametrize("edge", [15, 63])
def test_box_sizes_and_carries(ctx, oracle_lib, rng, frames, values, edge):
    """1 200-photon frames: 1.4e6 pairs and more (a small box), 2e7 and more (the
    largest), with sums that stay in the box's 32 bits and sums that leave them."""
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    shape = oracle_lib.big_mesh_shape(mq, edge)
    n = 1200 if frames < 100 else 400
    ph, off = random_frames(km, [n] * frames, rng, max_count=128 if values == "counts to 128" else 3,
                            integer=values.startswith("counts"))
    if values == "past 32 bits":
        ph[:, 3] *= 1000.0
    check(ctx, oracle_lib, ph, off, W.haar_rotations(frames, seed=6), shape, 1, 0, 0)


@pytest.mark.parametrize("frames", [3, 30])
@pytest.mark.parametrize("dmap", [0, 1])
def test_linear_with_the_box(ctx, oracle_lib, rng, frames, dmap):
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    for edge, max_count in ((31, 3), (63, 128)):
        shape = oracle_lib.big_mesh_shape(mq, edge)
        ph, off = random_frames(km, [1200] * frames, rng, max_count=max_count)
        check(ctx, oracle_lib, ph, off, W.haar_rotations(frames, seed=7), shape, dmap, 0, 1)


@pytest.mark.parametrize("dmap,i1,i2", MODES)
@pytest.mark.parametrize("pad", [0, 260], ids=["planned_by_the_kernel", "planner"])
@pytest.mark.parametrize("mult", [1000.0, 1234.5])
def test_frames_off_the_fast_path(ctx, oracle_lib, rng, dmap, i1, i2, pad, mult):
    """One batch of plain counts, a photon of value 0, a value above 128, real
    values, a rotation that leaves the mesh and one that shrinks."""
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    shape = oracle_lib.big_mesh_shape(mq, 31)
    sizes = [90, 77, 64, 33, 80, 70] + [3] * pad
    ph, off = random_frames(km, sizes, rng)
    ph[off[1] + 5, 3] = 0.0
    ph[off[2] + 6, 3] = 200.0
    ph[off[3]:off[4], 3] *= 0.73
    rot = W.haar_rotations(len(sizes), seed=9)
    rot[4] *= 1.4
    rot[5] *= 0.5
    check(ctx, oracle_lib, ph, off, rot, shape, dmap, i1, i2, mult)
