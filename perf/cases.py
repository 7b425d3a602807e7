"""The work that users of this framework have it do, as timed cases.

Every case goes through the public Python view of the C ABI
(incohautocorrelate_b200.capi) the way an evaluation, a simulation or a
training program calls it.  Inputs are synthetic, made on the GPU from the
seed alone, with the geometries and distributions of
incohautocorrelate_b200/workloads.py, bench.py and the tests:

* ``pairs``    photon lists -> uint64 pair mesh (one event of a live run, a
               batch of a rotated run, linear binning), nearest or linear on
               either level, single or double mapping;
* ``cq_map``   all pixel pairs of a mean-intensity map -> small C(q) mesh;
* ``ac1d_map`` the same pairs -> |q| histogram;
* ``cq_merge`` small C(q) mesh rotated by every frame into the cubic mesh;
* ``ac1d``     photon lists -> angular-averaged histogram, the reference's
               route choice per frame;
* ``simulate`` crystal -> emitters -> intensities -> Poisson photons -> lists;
* ``average``  averaged intensity and per-event means of loaded frames;
* ``ingest``   loaded frames -> masked, photonised sparse hit lists.

The mesh denoiser has its own sweep (bench.py --kernel denoise).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from incohautocorrelate_b200 import capi
from incohautocorrelate_b200 import workloads as W

PITCH = 75e-6

_ctx = None


def context():
    """One context per program, as a user keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = capi.Context(torch.cuda.current_device())
    return _ctx


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    two_panels = dict(ny=512, nx=1024, pitch_um=75.0, panels=2)
    return [
        # the smallest call: one event of a live run (128 x 128 detector, about 1 % of the pixels
        # hit) added to the 65^3 mesh by the allocation-free entry, for acquisition loops
        dict(name="pairs_one_event", kind="pairs", ny=128, nx=128, pitch_um=75.0, panels=1, frames=1,
             median=164.0, sigma=0.1, edge=63, double_map=True, first=0, second=0, route="static"),
        # the rotated correlator: a batch of 100 000 oriented frames of the two-panel detector,
        # cleared, binned and folded into the 201^3 mesh
        dict(name="pairs_rotated_batch", kind="pairs", frames=100_000, median=80.0, sigma=0.8, edge=199,
             double_map=True, first=0, second=0, route="device", **two_panels),
        # the same frames from pinned host lists, a batch of a long run whose mesh stays on the device
        dict(name="pairs_host_batch", kind="pairs", frames=20_000, median=80.0, sigma=0.8, edge=199,
             double_map=True, first=0, second=0, route="host", **two_panels),
        # linear binning of the rotated q (single mapping) of a short run on an odd-sized detector
        dict(name="pairs_linear", kind="pairs", ny=251, nx=245, pitch_um=150.0, panels=1, frames=3001,
             median=120.0, sigma=0.5, edge=127, double_map=False, first=0, second=1, route="device"),
        # the mean intensity's C(q) on the small mesh, once per evaluation: the two-panel detector,
        # nearest voxel, 201-edge small mesh
        dict(name="cq_map", kind="cq_map", edge=199, interp=0, **two_panels),
        # the same with linear interpolation on a small detector with ragged tiles
        dict(name="cq_map_linear", kind="cq_map", ny=244, nx=250, pitch_um=150.0, panels=1, edge=127, interp=1),
        # the angular-averaged evaluation's C(q): linear bins, as that run mode fixes them
        dict(name="ac1d_map", kind="ac1d_map", ny=512, nx=512, pitch_um=75.0, panels=1, bins=2048, interp=1),
        # the merge of the small C(q) mesh over the frames of a run
        dict(name="cq_merge", kind="cq_merge", edge=199, frames=10_000, interp=0),
        # the angular-averaged evaluation's frames: linear bins, route chosen per frame
        dict(name="ac1d_frames", kind="ac1d", frames=20_000, median=80.0, sigma=0.8, bins=2048, interp=1,
             **two_panels),
        # a chunk of the simulator: 5 x 5 x 8 emitters, 4 modes, Poisson photons, photon lists
        dict(name="simulate_frames", kind="simulate", det=512, cells_a=5, cells_b=5, cells_c=8, modes=4,
             frames=100, susa=0, squared=True, photons=0.02, fluorescence=1.0),
        # averaged intensity of a loaded batch without discretisation (analogue detector values)
        dict(name="average_frames", kind="average", ny=512, nx=1024, frames=300, threshold=0.2, step=0.0,
             masked=True),
        # sparse hit lists of a loaded batch: masked, thresholded, photonised, in pixel order
        dict(name="ingest_frames", kind="ingest", ny=512, nx=1024, frames=200, hits=0.01, threshold=0.5, step=1.0,
             masked=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(n):
    return int(n) | 1


def draw(rng):
    """One more case of the same ranges; a draw that would cost more than the
    largest listed case is shrunk."""
    kind = rng.choice(["pairs", "pairs", "cq_map", "ac1d_map", "cq_merge", "ac1d", "simulate", "average", "ingest"])
    if kind in ("pairs", "ac1d"):
        ny, nx = _log(rng, 100, 512), _log(rng, 100, 1024)
        median, sigma = float(_log(rng, 40, 300)), rng.choice([0.1, 0.5, 0.8])
        frames = _log(rng, 1, 100_000)
        per_frame = 0.5 * median * median * math.exp(2 * sigma * sigma)
        c = dict(kind=kind, ny=ny, nx=nx, pitch_um=float(round(75.0 * 512 / max(ny, nx), 2)), panels=1,
                 median=median, sigma=sigma)
        if kind == "ac1d":
            c.update(bins=_log(rng, 200, 4000), interp=rng.choice([0, 1, 1]))
            c["frames"] = max(1, min(frames, int(1.0e9 / per_frame)))
            return c
        first, second, dmap = rng.choice([(0, 0, True), (0, 0, True), (0, 0, False), (0, 1, False), (0, 1, True),
                                          (1, 0, True)])
        cost = 1 if not (first or second) else 10
        c.update(edge=_odd(_log(rng, 41, 201)), double_map=dmap, first=first, second=second,
                 route=rng.choice(["device", "device", "static", "host"]))
        c["frames"] = max(1, min(frames, int(1.2e9 / per_frame / cost)))
        return c
    if kind in ("cq_map", "ac1d_map"):
        interp = rng.choice([0, 1])
        most = 300_000 if kind == "ac1d_map" else (500_000 if interp == 0 else 80_000)
        ny, nx = _log(rng, 100, 700), _log(rng, 100, 1024)
        while ny * nx > most:
            ny, nx = int(ny * 0.9), int(nx * 0.9)
        c = dict(kind=kind, ny=ny, nx=nx, pitch_um=float(round(75.0 * 512 / max(ny, nx), 2)), panels=1, interp=interp)
        c.update(edge=_odd(_log(rng, 63, 253))) if kind == "cq_map" else c.update(bins=_log(rng, 200, 4000))
        return c
    if kind == "cq_merge":
        return dict(kind=kind, edge=_odd(_log(rng, 63, 201)), frames=_log(rng, 10, 15_000), interp=rng.choice([0, 0, 1]))
    if kind == "simulate":
        det, cells = rng.choice([128, 200, 256, 333, 512]), [rng.randint(2, 8) for _ in range(3)]
        susa, modes = rng.choice([0, 0, 0, 1]), rng.randint(1, 6)
        terms = det * det * cells[0] * cells[1] * cells[2] * modes * (2 * susa + 1) ** 2
        return dict(kind=kind, det=det, cells_a=cells[0], cells_b=cells[1], cells_c=cells[2], modes=modes,
                    frames=max(1, min(_log(rng, 1, 1000), int(4e10 / terms), int(6e7 / det / det))), susa=susa,
                    squared=rng.random() < 0.7, photons=rng.choice([0.005, 0.02, 0.1, 2.0]),
                    fluorescence=rng.choice([1.0, 1.0, 0.6]))
    if kind == "average":
        ny, nx = _log(rng, 100, 1024), _log(rng, 100, 1024)
        step = rng.choice([0.0, 0.0, 1.0, 0.73])
        return dict(kind=kind, ny=ny, nx=nx, frames=max(1, min(_log(rng, 1, 1000), int(2e8 / ny / nx))),
                    threshold=rng.choice([0.0, 0.2, 0.35]), step=step, masked=rng.random() < 0.7)
    ny, nx = _log(rng, 100, 1024), _log(rng, 100, 1024)
    return dict(kind=kind, ny=ny, nx=nx, frames=max(1, min(_log(rng, 1, 1000), int(1.5e8 / ny / nx))),
                hits=rng.choice([0.0002, 0.01, 0.1]), threshold=rng.choice([0.0, 0.5]), step=rng.choice([1.0, 0.73]),
                masked=rng.random() < 0.7)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _detector(case):
    """(pixel map in metres, k-map, MaxQ) of a flat detector normal to the beam."""
    two = case.get("panels", 1) == 2
    pm = W.flat_pixel_map(case["ny"], case["nx"], pitch=case["pitch_um"] * 1e-6, gap_x=2e-3 if two else 0.0,
                          gap_after=case["nx"] // 2 if two else None)
    km, mq = W.kmap_numpy(pm)
    return pm, km, mq


def _rotations(n, g):
    q = torch.randn((n, 4), generator=g, device="cuda", dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)
    return R.float().contiguous()


def _photons(case, km, g):
    """(float4 photon lists, int64 offsets) of frames whose photon number is
    Poisson around a log-normal mean; photons on one pixel add up, 5 % of the
    pixels are masked."""
    nf, npix = case["frames"], case["ny"] * case["nx"]
    lam = case["median"] * torch.exp(case["sigma"] * torch.randn(nf, generator=g, device="cuda", dtype=torch.float64))
    nph = torch.poisson(lam, generator=g).long()
    good = torch.nonzero(torch.rand(npix, generator=g, device="cuda") >= 0.05)[:, 0]
    pix = good[torch.randint(0, good.numel(), (int(nph.sum()),), generator=g, device="cuda")]
    frame = torch.repeat_interleave(torch.arange(nf, device="cuda"), nph)
    key, count = torch.unique(frame * npix + pix, return_counts=True)
    d_km = torch.from_numpy(km).cuda().view(-1, 3)
    ph = torch.cat([d_km[key % npix], count.float()[:, None]], 1).contiguous()
    if ph.shape[0] == 0:
        ph = torch.zeros((1, 4), device="cuda")
    off = torch.searchsorted(key, torch.arange(nf + 1, device="cuda") * npix)
    return ph, off.contiguous()


def _intensity(case, seed):
    """Mean intensity falling with the radius, 2 % noise, 5 % of the pixels masked."""
    return W.radial_mean_intensity(case["ny"], case["nx"], 0.3 * max(case["ny"], case["nx"]), 0.02, 0.05, seed)


def _zeros(n, dtype=torch.int64):
    return torch.zeros(n, dtype=dtype, device="cuda")


def prepare(case, seed):
    ctx, kind, g = context(), case["kind"], _generator(seed)
    s = {"case": case, "ctx": ctx, "stream": torch.cuda.current_stream().cuda_stream}
    if kind == "pairs":
        _, km, mq = _detector(case)
        s["photons"], s["offsets"] = _photons(case, km, g)
        s["rot"] = _rotations(case["frames"], g)
        shape = capi.big_mesh_shape(mq, case["edge"])
        s["S"] = shape.size_ab
        s["params"] = capi.sparse_params(shape, case["first"], case["second"], case["double_map"])
        s["half"] = _zeros(capi.half_mesh_words(s["S"]))
        if case["route"] == "device":
            s["full"] = _zeros(capi.full_mesh_words(s["S"]))
        if case["route"] == "host":
            for k in ("photons", "offsets", "rot"):
                s[k] = s[k].cpu().pin_memory()
    elif kind in ("cq_map", "ac1d_map"):
        _, km, mq = _detector(case)
        I = _intensity(case, seed)
        s["I"], s["km"] = torch.from_numpy(I).cuda(), torch.from_numpy(km).cuda()
        if kind == "cq_map":
            s["shape"] = sh = capi.small_cq_mesh_shape(mq, case["edge"])
            s["mult"] = capi.cq_small_multiplicator(I)
            s["out"] = _zeros(sh.size_ab * sh.size_ab * sh.size_c)
        else:
            s["shape"] = sh = capi.ac1d_shape(mq, case["bins"])
            s["mult"] = capi.ac1d_cq_multiplicator(I)
            s["out"] = _zeros(sh.size)
    elif kind == "cq_merge":
        # the small mesh of a coarse map of the two-panel detector's angular range
        det = dict(ny=128, nx=256, pitch_um=300.0, panels=1)
        _, km, mq = _detector(det)
        I = _intensity(det, seed)
        s["shape"] = sh = capi.small_cq_mesh_shape(mq, case["edge"])
        mult = capi.cq_small_multiplicator(I)
        small = _zeros(sh.size_ab * sh.size_ab * sh.size_c)
        ctx.cq_small(torch.from_numpy(I).cuda(), torch.from_numpy(km).cuda(), I.size, sh, 0, mult, small,
                     s["stream"], fast_size=det["nx"])
        h_small = small.cpu().numpy().view(np.uint64).astype(np.float64) / mult
        R = _rotations(case["frames"], g).cpu().numpy()
        MI = (0.5e-4 + 3.5e-4 * torch.rand(case["frames"], generator=g, device="cuda")).cpu().numpy()
        rw, s["mult"] = capi.cq_merge_weights(R, MI, h_small)
        s["small"], s["rw"] = torch.from_numpy(h_small).cuda(), torch.from_numpy(rw).cuda()
        s["big"] = _zeros(sh.size_ab ** 3)
    elif kind == "ac1d":
        _, km, mq = _detector(case)
        s["photons"], s["offsets"] = _photons(case, km, g)
        s["shape"] = sh = capi.ac1d_shape(mq, case["bins"])
        s["acc"] = _zeros(capi.ac1d_uw_words(sh))
        s["out"] = _zeros(sh.size, torch.float64)
    elif kind == "simulate":
        n, nf, nm = case["det"], case["frames"], case["modes"]
        pitch = PITCH * 512 / n
        pm = W.flat_pixel_map(n, n, pitch=pitch)
        km, _ = W.kmap_numpy(pm)
        cells = [case["cells_a"], case["cells_b"], case["cells_c"]]
        grid = np.stack(np.meshgrid(*[np.arange(c) - c / 2.0 + 0.5 for c in cells], indexing="ij"), -1)
        atoms = (4.0 * grid.reshape(-1, 3)).astype(np.float64)
        s["seed"], s["natoms"] = int(seed), len(atoms)
        s["atoms"] = torch.from_numpy(atoms.reshape(-1)).cuda()
        s["pm"] = torch.from_numpy((pm * np.float32(1e10)).astype(np.float32)).cuda()
        s["km"] = torch.from_numpy(km).cuda()
        s["em"] = _zeros((nf, nm, len(atoms), 4), torch.float32)
        s["count"] = _zeros(nf * nm, torch.int32)
        s["rot"] = _zeros((nf, 9), torch.float32)
        s["img"] = _zeros((nf, n * n), torch.float32)
        s["cap"] = int(nf * n * n * min(1.0, 1.5 * case["photons"])) + 20_000
        s["photons"] = _zeros((s["cap"], 4), torch.float32)
        s["offsets"] = _zeros(nf + 1)
        s["crystal"] = capi.CrystalParams(1, case["fluorescence"], 1, 1.0)
        us = pitch * 1e10 / (2 * case["susa"] + 1)
        s["sim"] = capi.SimParams(case["susa"], (C.c_double * 3)(us, 0, 0), (C.c_double * 3)(0, us, 0), 1.55,
                                  int(case["squared"]), 0)
        s["photon"] = capi.PhotonParams(case["photons"] * n * n, 1, 0.0, 1.0)
    elif kind == "average":
        npix, nf = case["ny"] * case["nx"], case["frames"]
        # analogue values: mostly near zero with a tail of photons
        u = torch.rand((nf, npix), generator=g, device="cuda")
        s["frames"] = (u.pow_(3.3).mul_(1.2)).contiguous()
        s["mask"] = (torch.rand(npix, generator=g, device="cuda") > 0.05).int() if case["masked"] else None
        s["sum"] = _zeros(npix, torch.float32) if case["step"] <= 0 else None
        s["discr"] = _zeros(npix) if case["step"] > 0 else None
        s["mean"] = _zeros(nf, torch.float32)
        s["counts"] = _zeros(nf, torch.float32) if case["step"] > 0 else None
        s["out"] = _zeros(npix, torch.float32)
    else:
        npix, nf = case["ny"] * case["nx"], case["frames"]
        _, km, _ = _detector(dict(case, pitch_um=75.0))
        s["km"] = torch.from_numpy(km).cuda()
        # electronic noise around zero, photons of about one unit on a share of the pixels
        v = 0.1 * torch.randn((nf, npix), generator=g, device="cuda")
        hit = torch.rand((nf, npix), generator=g, device="cuda") < case["hits"]
        s["frames"] = torch.where(hit, v + 1.0 + torch.floor(3 * torch.rand(v.shape, generator=g, device="cuda") ** 4), v)
        if case["threshold"] <= 0:  # counted photons: no noise
            s["frames"] = torch.where(hit, torch.round(s["frames"]), torch.zeros_like(v))
        s["mask"] = (torch.rand(npix, generator=g, device="cuda") > 0.05).int() if case["masked"] else None
        s["cap"] = int(1.5 * nf * npix * case["hits"]) + 20_000
        s["photons"] = _zeros((s["cap"], 4), torch.float32)
        s["offsets"] = _zeros(nf + 1)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, ctx, kind, st = s["case"], s["ctx"], s["case"]["kind"], s["stream"]
    if kind == "pairs":
        if case["route"] == "host":  # batches are added to a mesh that stays on the device
            ctx.sparse_ac_frames_host_to_device(s["photons"], s["offsets"], s["rot"], case["frames"], s["params"],
                                                s["half"], st)
            return s["half"]
        if case["route"] == "static":  # as are single events
            ctx.sparse_ac_batch_static(s["photons"], s["offsets"], s["rot"], case["frames"], s["params"], s["half"], st)
            return s["half"]
        s["half"].zero_()
        ctx.sparse_ac_batch(s["photons"], s["offsets"], s["rot"], case["frames"], s["params"], s["half"], st)
        s["full"].zero_()
        ctx.sparse_fold(s["half"], s["S"], s["full"], st)
        return s["full"]
    if kind == "cq_map":
        s["out"].zero_()
        ctx.cq_small(s["I"], s["km"], s["I"].numel(), s["shape"], case["interp"], s["mult"], s["out"], st,
                     fast_size=case["nx"])
        return s["out"]
    if kind == "ac1d_map":
        s["out"].zero_()
        ctx.ac1d_cq(s["I"], s["km"], s["I"].numel(), s["shape"], case["interp"], s["mult"], s["out"], st)
        return s["out"]
    if kind == "cq_merge":
        s["big"].zero_()
        ctx.cq_merge(s["small"], s["rw"], case["frames"], s["shape"], case["interp"], s["mult"], s["big"], st)
        return s["big"]
    if kind == "ac1d":
        s["acc"].zero_()
        ctx.ac1d_uw_batch(s["photons"], s["offsets"], case["frames"], case["ny"] * case["nx"], s["shape"],
                          case["interp"], s["acc"], stream=st)
        ctx.ac1d_uw_finish(s["acc"], s["shape"], s["out"], st)
        return s["out"]
    if kind == "simulate":
        nf, npix, na, nm = case["frames"], case["det"] ** 2, s["natoms"], case["modes"]
        ctx.crystal_emitters(s["atoms"], na, nf, nm, s["crystal"], s["seed"], s["em"], s["count"], s["rot"], None, st)
        ctx.simulate_intensity(s["pm"], npix, s["em"], s["count"], na, nm, nf, s["sim"], s["img"], st)
        ctx.simulate_photons(s["img"], npix, nf, 0, s["photon"], s["seed"] + 1, st)
        ctx.sparsify_frames(s["img"], None, s["km"], npix, nf, 0.0, 1.0, 1, s["photons"], s["cap"], s["offsets"], st,
                            want_total=False)
        return {"images": s["img"], "photons": s["photons"], "offsets": s["offsets"], "rotations": s["rot"]}
    if kind == "average":
        npix, nf = case["ny"] * case["nx"], case["frames"]
        for buf in (s["sum"], s["discr"]):
            if buf is not None:
                buf.zero_()
        ctx.average_frames(s["frames"], npix, nf, s["mask"], case["threshold"], case["step"], s["sum"], s["discr"],
                           s["mean"], s["counts"], st)
        ctx.average_finish(s["sum"], s["discr"], npix, nf, s["out"], st)
        return {"intensity": s["out"], "means": s["mean"], "counts": s["counts"]}
    ctx.sparsify_frames(s["frames"], s["mask"], s["km"], case["ny"] * case["nx"], case["frames"], case["threshold"],
                        case["step"], 1, s["photons"], s["cap"], s["offsets"], st, want_total=False)
    return {"photons": s["photons"], "offsets": s["offsets"]}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _expected_pairs(case):
    """(photons, unordered pairs with self pairs) expected in the frames of a case."""
    m, s2 = case["median"], case["sigma"] ** 2
    mean, square = m * math.exp(0.5 * s2), m * m * math.exp(2 * s2)
    return case["frames"] * mean, case["frames"] * (0.5 * square + mean)


def work(case):
    kind = case["kind"]
    if kind == "pairs":
        photons, pairs = _expected_pairs(case)
        S = case["edge"] + 2
        half = 8.0 * S * S * (S + 1) / 2
        inputs = 16.0 * photons + 44.0 * case["frames"]
        # difference 3, norm 5, scale 3, rotation 15; every voxel touched is read and written
        mesh = 16.0 * min(pairs, half / 8) if case["route"] != "device" else 8.0 * S ** 3
        return {"bytes": inputs + mesh, "flops": 26.0 * pairs}
    if kind in ("cq_map", "ac1d_map"):
        n = float(case["ny"] * case["nx"])
        pairs = n * (n + 1) / 2
        if kind == "cq_map":
            e = case["edge"] + 2
            return {"bytes": 16.0 * n + 8.0 * e * e * (e / 8.0), "flops": 12.0 * pairs}
        return {"bytes": 16.0 * n + 8.0 * case["bins"], "flops": 11.0 * pairs}
    if kind == "cq_merge":
        e = case["edge"] + 2
        voxels = 0.5 * e * e * (e / 8.0)
        return {"bytes": 8.0 * e ** 3 + 8.0 * voxels + 40.0 * case["frames"], "flops": 16.0 * voxels * case["frames"]}
    if kind == "ac1d":
        photons, pairs = _expected_pairs(case)
        return {"bytes": 16.0 * photons + 8.0 * case["frames"] + 8.0 * case["bins"], "flops": 11.0 * pairs}
    if kind == "simulate":
        npix, nf = case["det"] ** 2, case["frames"]
        terms = float(npix) * case["cells_a"] * case["cells_b"] * case["cells_c"] * case["modes"] * nf
        terms *= (2 * case["susa"] + 1) ** 2 * case["fluorescence"]
        photons = npix * nf * min(1.0, case["photons"])
        return {"bytes": 4.0 * npix * nf + 16.0 * photons + 24.0 * npix, "flops": 10.0 * terms}
    if kind == "average":
        npix, nf = float(case["ny"] * case["nx"]), case["frames"]
        return {"bytes": 4.0 * npix * nf + 12.0 * npix + 4.0 * nf, "flops": 2.0 * npix * nf}
    npix, nf = float(case["ny"] * case["nx"]), case["frames"]
    return {"bytes": 4.0 * npix * nf + 16.0 * npix + 16.0 * case["hits"] * npix * nf, "flops": 2.0 * npix * nf}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _exact_average(case, seed):
    s = prepare(case, seed)
    mask = 1.0 if s["mask"] is None else s["mask"].double()
    total = torch.zeros(case["ny"] * case["nx"], dtype=torch.float64, device="cuda")
    means, counts = [], []
    for frame in s["frames"]:
        v = frame.double() * mask
        on = v >= float(np.float32(case["threshold"]))
        if case["step"] > 0:
            thr, step = (float(np.float32(case[k])) for k in ("threshold", "step"))
            v = torch.where(on, torch.ceil((v - thr) / step), torch.zeros_like(v))
            counts.append(v.sum())
        elif case["threshold"] > 0:
            v = torch.where(on, v, torch.zeros_like(v))
        total += v
        means.append(v.sum() / v.numel())
    return {"intensity": total / case["frames"], "means": torch.stack(means),
            "counts": torch.stack(counts) if counts else None}


def _exact_ac1d(case, seed):
    """Unordered pairs k >= j with a factor 2, bins and weights in 64 bits; the
    frames whose hits reach 0.75 % of the pixels count the self pairs once."""
    if _expected_pairs(case)[1] > 3e8:
        return None
    s = prepare(case, seed)
    sh, off = s["shape"], s["offsets"].tolist()
    out = torch.zeros(sh.size + 2, dtype=torch.float64, device="cuda")
    for f in range(case["frames"]):
        p = s["photons"][off[f]:off[f + 1]].double()
        n = p.shape[0]
        once = n / (case["ny"] * case["nx"]) >= 0.0075
        j, k = torch.triu_indices(n, n, device="cuda")
        q = (p[j, :3] - p[k, :3]).norm(dim=1)
        v = 2.0 * p[j, 3] * p[k, 3]
        if once:
            v = torch.where(j == k, v / 2, v)
        keep = q <= float(sh.max_q)
        q, v = q[keep] / float(sh.dq_per_step), v[keep]
        if case["interp"] == 0:
            out.index_add_(0, torch.floor(q + 0.5).long(), v)
        else:
            b = torch.floor(q).long()
            out.index_add_(0, b, v * (1 - (q - b)))
            out.index_add_(0, b + 1, v * (q - b))
    return out[:sh.size]


def exact(case, seed):
    if case["kind"] == "average":
        return _exact_average(case, seed)
    if case["kind"] == "ac1d":
        return _exact_ac1d(case, seed)
    # meshes, histograms, photon images and lists hold whole numbers and copies of inputs: compared as they are
    return None
