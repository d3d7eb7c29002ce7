"""Timed cases of the photon mapper, each through the public entry points of
cuda-photon-mapper_gb300/photonmap.py (the binding of include/pm.h).

A case is a dict of plain values with a "kind":

  legacy   one frame of the reference's voxel mapper (emission + render)
  frame    one physically based frame: emission, kd build, render
  render   the render of an unchanged scene's maps (a still or a moved camera)
  points   kd build over a loaded point set + k-NN queries on it
  knn      k-NN queries on a built map
  noalloc  pm_knn_noalloc: build + queries without device allocation
  radius   the reference's record-list radius gather on a built map
  cache    one online frame of the radiance cache: training + cached render
  batch    one replayed frame of many scenes
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-photon-mapper_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import photonmap  # noqa: E402

# The box of every preset: [-0.5, 0.5] x [0, 1] x [-0.5, 0.5].
_BOX_LO = (-0.5, 0.0, -0.5)


def listed():
    return [
        # the reference's own window: 512 x 512 with the 'i' and 'p' keys on
        {"name": "legacy_512_media", "kind": "legacy", "width": 512, "height": 512, "interpolate": True, "media": True},
        # the same frame loop at thumbnail size with both keys off: the smallest frame there is
        {"name": "legacy_thumb", "kind": "legacy", "width": 161, "height": 119, "interpolate": False, "media": False},
        # the small benchmark preset, a whole frame: interactive use
        {"name": "frame_preset1", "kind": "frame", "preset": 1, "surface": 100000, "volume": 100000,
         "width": 512, "height": 512, "k": 64, "radius": 0.1},
        # a preview frame at a ragged size with unequal maps, k not a multiple of 32
        {"name": "frame_preview", "kind": "frame", "preset": 2, "surface": 123457, "volume": 54321,
         "width": 333, "height": 217, "k": 50, "radius": 0.08},
        # the headline workload: 64 spheres, heterogeneous medium, 8M + 8M photons
        {"name": "frame_preset3", "kind": "frame", "preset": 3, "surface": 8000000, "volume": 8000000,
         "width": 1920, "height": 1080, "k": 128, "radius": 0.05},
        # the medium benchmark preset with its maps kept: the camera's frame over unchanged photons
        {"name": "render_preset2", "kind": "render", "preset": 2, "surface": 1000000, "volume": 1000000,
         "width": 1024, "height": 1024, "k": 100, "radius": 0.05},
        # a small loaded point set, its tree and a few thousand queries: latency and launches
        {"name": "points_small", "kind": "points", "n": 20011, "nq": 4099, "k": 16, "radius": 0.1},
        # many queries near the points of a built map, in no particular order
        {"name": "knn_1m", "kind": "knn", "n": 1000000, "nq": 262144, "k": 100, "radius": 0.05},
        # the allocation-free entry near its largest point count
        {"name": "noalloc_100k", "kind": "noalloc", "n": 100000, "nq": 32768, "k": 32, "radius": 0.1},
        # the reference's radius gather over a surface map
        {"name": "radius_500k", "kind": "radius", "n": 500000, "nq": 131072, "sq_radius": 0.0004, "exposure": 50.0},
        # the radiance cache's online frame on the medium preset (2^20 targets, 8 Adam steps, cached render)
        {"name": "cache_preset2", "kind": "cache", "preset": 2, "surface": 1000000, "volume": 1000000,
         "width": 1024, "height": 1024, "k": 100, "radius": 0.05, "samples": 1 << 20, "batch": 1 << 17, "log2_table": 19},
        # scenes 8 .. 13 of the batched workload replayed as one graph
        {"name": "batch_6", "kind": "batch", "first": 8, "scenes": 6, "max_res": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["legacy", "frame", "frame", "render", "points", "knn", "noalloc", "radius", "cache", "batch"])
    if kind == "legacy":
        return {"kind": kind, "width": _log(rng, 64, 1024), "height": _log(rng, 64, 1024),
                "interpolate": rng.random() < 0.5, "media": rng.random() < 0.5}
    if kind in ("frame", "render", "cache"):
        preset = rng.choice([1, 2, 3] if kind == "frame" else [1, 2])
        c = {"kind": kind, "preset": preset, "surface": _log(rng, 20000, 2000000),
             "volume": _log(rng, 20000, 2000000), "width": _log(rng, 100, 1000), "height": _log(rng, 100, 800),
             "k": rng.choice([16, 32, 50, 64, 100, 128]), "radius": rng.choice([0.05, 0.08])}
        if kind == "cache":
            c["batch"] = 128 * _log(rng, 64, 1024)
            c["samples"] = min(1 << 20, c["batch"] * rng.randint(1, 8))
            c["log2_table"] = rng.randint(15, 19)
        return c
    if kind == "points":
        return {"kind": kind, "n": _log(rng, 1000, 2000000), "nq": _log(rng, 1000, 65536),
                "k": _log(rng, 1, 128), "radius": rng.choice([0.05, 0.1])}
    if kind == "knn":
        return {"kind": kind, "n": _log(rng, 20000, 4000000), "nq": _log(rng, 500, 262144),
                "k": _log(rng, 1, 128), "radius": rng.choice([0.05, 0.1])}
    if kind == "noalloc":
        return {"kind": kind, "n": _log(rng, 1000, 131072), "nq": _log(rng, 500, 65536),
                "k": _log(rng, 1, 128), "radius": rng.choice([0.05, 0.1])}
    if kind == "radius":
        return {"kind": kind, "n": _log(rng, 20000, 2000000), "nq": _log(rng, 1000, 131072),
                "sq_radius": rng.choice([0.0001, 0.0004, 0.0009]), "exposure": rng.choice([1.0, 50.0])}
    return {"kind": kind, "first": rng.randint(0, 58), "scenes": rng.randint(2, 6), "max_res": rng.choice([256, 512])}


def _stream():
    return torch.cuda.current_stream().cuda_stream


class _State:
    """What a case's program keeps: its context and its buffers."""


def _context():
    return photonmap.Context(torch.cuda.current_device())


def _scene(case, seed):
    sc, cf = photonmap.preset(case["preset"], 0x5EED0000 + int(seed))
    cf.surface_photons = case["surface"]
    cf.volume_photons = case["volume"]
    cf.width, cf.height = case["width"], case["height"]
    cf.k = case["k"]
    cf.radius = case["radius"]
    return sc, cf


def _image(st, width, height):
    st.rad = torch.zeros((height, width, 4), dtype=torch.float32, device="cuda")
    st.rgba = torch.zeros((height, width, 4), dtype=torch.uint8, device="cuda")


def _points(n, nq, seed):
    """n points in the preset box -- a third on its walls, a third uniform, a
    third in clusters, as photon maps hold them -- with unit directions and
    positive fluxes, and nq queries beside points and anywhere in the box."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)

    def u(*s):
        return torch.rand(*s, generator=g, device="cuda")

    lo = torch.tensor(_BOX_LO, device="cuda")
    p = u(n, 3)
    wall = torch.arange(n, device="cuda") % 3 == 0
    axis = torch.randint(0, 3, (n,), generator=g, device="cuda")
    side = torch.randint(0, 2, (n,), generator=g, device="cuda").float()
    on = wall[:, None] & (torch.arange(3, device="cuda")[None, :] == axis[:, None])
    p = torch.where(on, side[:, None], p)
    centre = u(64, 3) * 0.8 + 0.1
    which = torch.randint(0, 64, (n,), generator=g, device="cuda")
    cl = centre[which] + 0.03 * torch.randn((n, 3), generator=g, device="cuda")
    p = torch.where((torch.arange(n, device="cuda") % 3 == 2)[:, None], cl.clamp(0.0, 1.0), p)
    pos = torch.zeros((n, 4), device="cuda")
    pos[:, :3] = p + lo
    d = torch.randn((n, 3), generator=g, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    # octahedral direction, two snorm16 values in the flux record's last word
    l1 = d.abs().sum(dim=1)
    px, py = d[:, 0] / l1, d[:, 1] / l1
    qx = (1 - py.abs()) * torch.where(px >= 0, 1.0, -1.0)
    qy = (1 - px.abs()) * torch.where(py >= 0, 1.0, -1.0)
    px, py = torch.where(d[:, 2] < 0, qx, px), torch.where(d[:, 2] < 0, qy, py)
    ix = torch.round(px.clamp(-1, 1) * 32767).to(torch.int32) & 0xFFFF
    iy = torch.round(py.clamp(-1, 1) * 32767).to(torch.int32) & 0xFFFF
    pw = torch.zeros((n, 4), device="cuda")
    pw[:, :3] = (0.2 + 0.8 * u(n, 3)) / n
    pw[:, 3] = (ix | (iy << 16)).view(torch.float32)
    q = torch.zeros((nq, 4), device="cuda")
    near = torch.randint(0, n, (nq,), generator=g, device="cuda")
    q[:, :3] = pos[near, :3] + 0.004 * torch.randn((nq, 3), generator=g, device="cuda")
    free = torch.arange(nq, device="cuda") % 4 == 3
    q[:, :3] = torch.where(free[:, None], u(nq, 3) + lo, q[:, :3])
    nrm = torch.zeros((nq, 4), device="cuda")
    v = torch.randn((nq, 3), generator=g, device="cuda")
    nrm[:, :3] = v / v.norm(dim=1, keepdim=True)
    return pos, pw, q, nrm


def _loaded_map(case, st, pos, pw):
    sc, cf = photonmap.preset(1)
    cf.surface_photons, cf.volume_photons = case["n"], 0
    st.ctx = _context()
    st.ctx.set_scene(sc, cf)
    st.ctx.set_photons(photonmap.MAP_SURFACE, pos.cpu().numpy(), pw.cpu().numpy())
    st.ctx.build(_stream())


class _Device:
    """A library-owned device buffer as a tensor (no copy)."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    st = _State()
    st.case, st.kind = case, kind
    if kind == "legacy":
        st.ctx = _context()
        rng = np.random.RandomState(int(seed) & 0x7FFFFFFF)
        st.time = float(rng.uniform(0.0, 6.0))
        st.flags = (photonmap.PM_LEGACY_INTERPOLATE if case["interpolate"] else 0) | \
                   (photonmap.PM_LEGACY_MEDIA if case["media"] else 0)
        st.ctx.legacy_init_random(_stream())
        w, h = case["width"], case["height"]
        st.pos = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        st.rgb = torch.zeros((h, w, 3), dtype=torch.float32, device="cuda")
    elif kind in ("frame", "render", "cache"):
        sc, cf = _scene(case, seed)
        st.ctx = _context()
        st.ctx.set_scene(sc, cf)
        _image(st, cf.width, cf.height)
        if kind != "frame":
            st.ctx.emit(_stream())
            st.ctx.build(_stream())
        if kind == "cache":
            st.ctx.cache_enable(train_samples=case["samples"], batch=case["batch"], log2_table=case["log2_table"],
                                seed=0x5EED0004 + int(seed))
            st.weights = np.zeros(photonmap.CACHE_WEIGHTS, np.float32)
            st.ctx.cache_train(2, _stream())
    elif kind in ("points", "knn", "noalloc"):
        pos, pw, st.q, _ = _points(case["n"], case["nq"], seed)
        st.idx = torch.zeros((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        st.d2 = torch.zeros((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
        if kind == "noalloc":
            st.pos = pos
            st.lib = photonmap.load()
        else:
            _loaded_map(case, st, pos, pw)
    elif kind == "radius":
        pos, pw, st.q, st.nrm = _points(case["n"], case["nq"], seed)
        _loaded_map(case, st, pos, pw)
        st.out = torch.zeros((case["nq"], 4), dtype=torch.float32, device="cuda")
    else:
        scenes, cfgs = [], []
        for i in range(case["first"], case["first"] + case["scenes"]):
            # another seed gives other spheres, media and photons; the sizes stay the workload's
            _, size = photonmap.batch_scene(i, 0x5EED0005)
            sc, cf = photonmap.batch_scene(i, 0x5EED0005 + int(seed))
            cf.width, cf.height = min(size.width, case["max_res"]), min(size.height, case["max_res"])
            cf.surface_photons, cf.volume_photons, cf.k = size.surface_photons, size.volume_photons, size.k
            scenes.append(sc)
            cfgs.append(cf)
        st.ctx = _context()
        st.batch = photonmap.Batch(st.ctx, scenes, cfgs)
        s = torch.cuda.Stream()
        st.batch.frame(s.cuda_stream)
        s.synchronize()
        st.batch.capture(s.cuda_stream)
        s.synchronize()
        st.images = []
        for i, cf in enumerate(cfgs):
            rad, rgba = st.batch.image_ptrs(i)
            st.images.append(torch.as_tensor(_Device(rad, (cf.height, cf.width, 4), "<f4", st.batch), device="cuda"))
            st.images.append(torch.as_tensor(_Device(rgba, (cf.height, cf.width, 4), "|u1", st.batch), device="cuda"))
    return st


def run(st):
    case, kind, s = st.case, st.kind, _stream()
    if kind == "legacy":
        st.ctx.legacy_emit(st.time, st.flags, s)
        st.ctx.legacy_render(st.pos.data_ptr(), case["width"], case["height"], st.time, st.flags, st.rgb.data_ptr(), s)
        return {"pos": st.pos, "rgb": st.rgb}
    if kind == "frame":
        st.ctx.emit(s)
        st.ctx.build(s)
        st.ctx.render(st.rad.data_ptr(), st.rgba.data_ptr(), s)
        return {"radiance": st.rad, "rgba": st.rgba}
    if kind == "render":
        st.ctx.render(st.rad.data_ptr(), st.rgba.data_ptr(), s)
        return {"radiance": st.rad, "rgba": st.rgba}
    if kind == "cache":
        st.ctx.cache_train(1, s)
        st.ctx.render_cached(st.rad.data_ptr(), st.rgba.data_ptr(), 0, s)
        st.ctx.lib.pm_cache_get_params(st.ctx.h, st.weights.ctypes.data, None, None)
        return {"radiance": st.rad, "rgba": st.rgba, "weights": st.weights}
    if kind == "points":
        st.ctx.build(s)
    if kind in ("points", "knn"):
        st.ctx.knn(photonmap.MAP_SURFACE, st.q.data_ptr(), case["nq"], case["k"], case["radius"], st.idx.data_ptr(),
                   st.d2.data_ptr(), s)
        return {"idx": st.idx, "d2": st.d2}
    if kind == "noalloc":
        r = st.lib.pm_knn_noalloc(st.pos.data_ptr(), case["n"], st.q.data_ptr(), case["nq"], case["k"], case["radius"],
                                  st.idx.data_ptr(), st.d2.data_ptr(), s)
        if r != photonmap.PM_OK:
            raise photonmap.PMError("pm_knn_noalloc: %d" % r)
        return {"idx": st.idx, "d2": st.d2}
    if kind == "radius":
        st.ctx.radius_gather(photonmap.MAP_SURFACE, st.q.data_ptr(), st.nrm.data_ptr(), case["nq"], case["sq_radius"],
                             case["exposure"], st.out.data_ptr(), s)
        return {"out": st.out}
    st.batch.launch(s)
    return {"images": st.images}


# Per-unit work of the paths. A photon path and its interactions: one test per
# sphere and plane (about 16 operations each) and about 150 operations of
# sampling; an estimate: k records weighted and summed (about 20 operations
# each). Bytes are inputs and outputs only: records and trees that a frame
# makes on the way are counted once, as they are its maps.
_GATHERS_PER_PIXEL = {1: 45, 2: 40, 3: 10}
_SPHERES = {1: 2, 2: 8, 3: 64}


def _frame_work(case, emission):
    px = case["width"] * case["height"]
    rec = case["surface"] + case["volume"]
    gathers = px * _GATHERS_PER_PIXEL[case["preset"]]
    flops = gathers * case["k"] * 20.0
    if emission:
        flops += 4.0 * case["volume"] * 4 * (150 + 16 * (_SPHERES[case["preset"]] + 5))
    return {"bytes": 32.0 * rec + 20.0 * px, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "legacy":
        px = case["width"] * case["height"]
        return {"bytes": 16.0 * px + 32 ** 3 * 12 + 10000 * 16,
                "flops": 10000 * 5 * 2 * (36 * 8 + 100) + px * (300.0 + (200 if case["media"] else 0))}
    if kind in ("frame", "render"):
        return _frame_work(case, kind == "frame")
    if kind == "cache":
        w = _frame_work(case, False)
        q = case["width"] * case["height"] * _GATHERS_PER_PIXEL[case["preset"]]
        w["bytes"] += 16 * 2.0 ** case["log2_table"] * 28
        w["flops"] = case["samples"] * (case["k"] * 20.0 + 3 * 34816) + q * (34816.0 + 16 * 8 * 4)
        return w
    if kind in ("points", "knn", "noalloc"):
        n, nq, k = case["n"], case["nq"], case["k"]
        flops = nq * k * 10.0 + (0 if kind == "knn" else n * math.log2(max(n, 2)) * 4)
        return {"bytes": 16.0 * n + 16.0 * nq + 8.0 * nq * k, "flops": flops}
    if kind == "radius":
        inside = case["n"] * 4.19 * case["sq_radius"] ** 1.5
        return {"bytes": 32.0 * case["n"] + 48.0 * case["nq"], "flops": case["nq"] * (50 + inside * 30.0)}
    bytes_, flops = 0.0, 0.0
    for i in range(case["first"], case["first"] + case["scenes"]):
        sc, cf = photonmap.batch_scene(i, 0x5EED0005)
        px = min(cf.width, case["max_res"]) * min(cf.height, case["max_res"])
        rec = cf.surface_photons + cf.volume_photons
        bytes_ += 32.0 * rec + 20.0 * px
        flops += px * 40 * cf.k * 20.0 + 4.0 * cf.volume_photons * 4 * (150 + 16 * (sc.num_spheres + 5))
    return {"bytes": bytes_, "flops": flops}


def _directions(word):
    b = word.view(torch.int32)

    def snorm(v):
        v = v & 0xFFFF
        return torch.where(v >= 0x8000, v - 0x10000, v).double() / 32767.0

    px, py = snorm(b), snorm(b >> 16)
    pz = 1.0 - px.abs() - py.abs()
    qx = (1 - py.abs()) * torch.where(px >= 0, 1.0, -1.0)
    qy = (1 - px.abs()) * torch.where(py >= 0, 1.0, -1.0)
    px, py = torch.where(pz < 0, qx, px), torch.where(pz < 0, qy, py)
    d = torch.stack((px, py, pz), dim=1)
    return d / d.norm(dim=1, keepdim=True)


def exact(case, seed):
    """Brute force in 64 bits over the same points. The images and the
    network's weights have no such value: they follow random paths, whose
    choices another precision would make differently."""
    kind = case["kind"]
    if kind not in ("points", "knn", "noalloc", "radius") or case["n"] * case["nq"] > 7e10:
        return None
    pos, pw, q, nrm = _points(case["n"], case["nq"], seed)
    p = pos[:, :3].double()
    rows = max(1, min(case["nq"], (1 << 27) // case["n"]))
    outs = []
    if kind == "radius":
        d, flux = _directions(pw[:, 3]), pw[:, :3].double()
    r2 = float(np.float32(case["radius"]) ** 2) if kind != "radius" else float(np.float32(case["sq_radius"]))
    for a in range(0, case["nq"], rows):
        x = q[a:a + rows, :3].double()
        s = sum((x[:, None, i] - p[None, :, i]) ** 2 for i in range(3))
        if kind == "radius":
            w = -(nrm[a:a + rows, :3].double() @ d.t()).clamp(max=0.0) * (1.0 - s.sqrt()) / float(np.float32(case["exposure"]))
            e = torch.where(s <= r2, w, 0.0) @ flux
            outs.append(torch.cat((e, torch.zeros_like(e[:, :1])), dim=1))
        else:
            kk = min(case["k"], case["n"])
            t = torch.topk(s, kk, dim=1, largest=False, sorted=True).values.clamp(max=r2)
            outs.append(torch.cat((t, torch.full((len(t), case["k"] - kk), r2, dtype=t.dtype, device=t.device)), dim=1))
    got = torch.cat(outs)
    return {"out": got} if kind == "radius" else {"idx": None, "d2": got}
