"""Host threads that share a context, each on its own stream: launches whose
kernels are the same and whose shared memory differs (the pair kernel's box by
mesh edge, the AC1D histograms by size) must not disturb one another."""
import threading

import numpy as np
import pytest

from helpers import random_frames, small_detector, to_capi_shape

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _run(works, rounds=300):
    """Every work once alone, then all of them `rounds` times side by side."""
    import torch
    want = []
    for once, out in works:
        once(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(out.clone())
        out.zero_()
    torch.cuda.synchronize()
    errors = []

    def loop(once):
        try:
            stream = torch.cuda.Stream()
            for _ in range(rounds):
                once(stream.cuda_stream)
            stream.synchronize()
        except Exception as e:  # reported by the test
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(once,)) for once, _ in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]
    for (_, out), w in zip(works, want):
        np.testing.assert_array_equal(out.cpu().numpy(), rounds * w.cpu().numpy())


def test_pair_meshes_of_different_edges(ctx, oracle_lib, rng):
    import torch
    from incohautocorrelate_b200 import capi
    from incohautocorrelate_b200 import workloads as W
    _, km, mq = small_detector()
    ph, off = random_frames(km, [40] * 8, rng)
    d = _dev(ph), _dev(off.astype(np.int64)), _dev(W.haar_rotations(8, seed=3).astype(np.float32))
    works = []
    for edge in (31, 63, 21, 41, 31, 63, 27, 35):
        shape = to_capi_shape(oracle_lib.big_mesh_shape(mq, edge))
        p, half = capi.sparse_params(shape), torch.zeros(capi.half_mesh_words(shape.size_ab), dtype=torch.int64, device="cuda")
        works.append((lambda s, p=p, half=half: ctx.sparse_ac_batch(*d, 8, p, half, s), half))
    _run(works, rounds=3000)


@pytest.mark.parametrize("interp", [0, 1])
def test_ac1d_shapes_of_different_sizes(ctx, rng, interp):
    import torch
    from incohautocorrelate_b200 import capi
    ny, nx = 16, 32
    _, km, mq = small_detector(ny, nx, 6e-4)
    ph, off = random_frames(km, [40] * 8, rng)
    d = _dev(ph), _dev(off.astype(np.int64))
    I, k = _dev(rng.uniform(0.05, 1.5, ny * nx).astype(np.float32)), _dev(km)
    rows = _dev(np.arange(64, dtype=np.int32))
    works = []
    for size in (1000, 7000):
        sh = capi.ac1d_shape(mq, size)
        acc = torch.zeros(capi.ac1d_uw_words(sh), dtype=torch.int64, device="cuda")
        works.append((lambda s, sh=sh, acc=acc: ctx.ac1d_uw_batch(*d, 8, ny * nx, sh, interp, acc, route=1, stream=s), acc))
        hist = torch.zeros(sh.size, dtype=torch.int64, device="cuda")
        works.append((lambda s, sh=sh, hist=hist: ctx.ac1d_cq(I, k, ny * nx, sh, interp, 1000.0, hist, s), hist))
        part = torch.zeros(sh.size, dtype=torch.int64, device="cuda")
        works.append((lambda s, sh=sh, part=part: ctx.ac1d_cq_rows(I, k, ny * nx, rows, 64, sh, interp, 1000.0, part, s), part))
    _run(works)
