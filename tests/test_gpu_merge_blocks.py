"""C(q) merge over the edges of its voxel blocks and frame pairs, bit for bit
against the oracle: odd frame counts on both sides of a chunk, meshes that are
not a multiple of a block, rotations that leave the mesh, values past 2^52."""
import numpy as np
import pytest

from helpers import to_capi_shape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("edge,frames,stretch,mult", [
    (5, 1, 1.0, 1e4), (9, 2, 1.0, 1e4), (9, 3, 1.6, 1e4), (21, 127, 1.0, 1e3), (21, 129, 1.3, 1e3), (11, 5, 1.0, 1e15),
])
def test_merge_blocks(ctx, oracle_lib, rng, interp, edge, frames, stretch, mult):
    import torch
    from incohautocorrelate_b200 import workloads as W
    o = oracle_lib
    s = o.small_cq_mesh_shape(np.array([1.0, 0.9, 0.4], np.float32), edge - 2)
    ab, sc = s.size_ab, s.size_c
    small = rng.uniform(0.0, 30.0, ab * ab * sc)
    small[rng.random(small.size) < 0.6] = 0.0
    rw = np.zeros((frames, 10), np.float32)
    rw[:, :9] = W.haar_rotations(frames, seed=5).reshape(frames, 9) * np.float32(stretch)
    rw[:, 9] = rng.uniform(0.1, 2.0, frames)
    want = np.zeros(ab ** 3, np.uint64)
    lost = o.lib().iaco_cq_merge(o.p(small), o.p(rw), frames, s, interp, mult, 0, small.size, o.p(want))
    out = torch.zeros(want.size, dtype=torch.int64, device="cuda")
    ctx.cq_merge(torch.from_numpy(small).cuda(), torch.from_numpy(rw).cuda(), frames, to_capi_shape(s), interp, mult, out)
    skipped = ctx.check()  # counts lost values that are not 0; the oracle counts every lost corner
    assert skipped <= lost and (skipped == lost or interp == 1)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("interp", [0, 1])
def test_merge_coordinates_past_the_floats(ctx, oracle_lib, rng, interp):
    """A rotation whose products overflow to infinity: its voxels are counted as
    lost, and the cubic mesh holds the other frames' alone."""
    import torch
    from incohautocorrelate_b200 import workloads as W
    o = oracle_lib
    s = o.small_cq_mesh_shape(np.array([1.0, 0.9, 0.4], np.float32), 11)
    small = rng.uniform(0.5, 30.0, s.size_ab * s.size_ab * s.size_c)
    rw = np.zeros((3, 10), np.float32)
    rw[:, :9] = W.haar_rotations(3, seed=5).reshape(3, 9)
    rw[1, :3] = 3e38, 0, 0
    rw[:, 9] = 1.0
    want = np.zeros(s.size_ab ** 3, np.uint64)
    lost = o.lib().iaco_cq_merge(o.p(small), o.p(rw), 3, s, interp, 1e3, 0, small.size, o.p(want))
    out = torch.zeros(want.size, dtype=torch.int64, device="cuda")
    ctx.cq_merge(torch.from_numpy(small).cuda(), torch.from_numpy(rw).cuda(), 3, to_capi_shape(s), interp, 1e3, out)
    skipped = ctx.check()
    assert 0 < skipped <= lost and (skipped == lost or interp == 1)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)
