"""The work that programs have this framework do, as cases that can be timed.

Each case is one call (or the few calls of one step) of the public entry
points, as a program makes them: ray queries through the C ABI without
allocation (``rmcuda_trace_noalloc``) and on the resident scene
(``Backend.trace``), single frames from host scenes (``Backend.render``) and of
resident scenes, the plain path tracer and the ReSTIR chain with its denoiser,
a frame of an animated world, loading a scene, a batch of uneven images, and a
material-fit step (forward frame and its adjoint) on both chains.

Sizes: the Cornell box, the 1,028,098-triangle icosphere field, the animated
sequence, the batch of uneven fields and the inverse-rendering scene are those
of ``raymotion_b200.scenes``; the small, odd ones are generic.  A case holds
``kind`` and that kind's sizes.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import raymotion_b200 as rb
from raymotion_b200 import _abi, objects
from raymotion_b200.scene import with_materials
from raymotion_b200.scenes import (PLAIN_FLAGS, AnimatedSequence, cornell_box, icosphere_field, inverse_scene,
                                   sized_field)

FAR = 200.0  # length of a query ray: beyond every scene


def listed():
    return [
        # picking and visibility in a small scene by a caller that may not allocate: latency and launches
        dict(name="query_noalloc_small", kind="noalloc", tris=1000, rays=4096, any_hit=False),
        # closest hits of incoherent rays in a large resident scene (light probes, lidar)
        dict(name="query_closest_large", kind="trace", tris=512000, rays=1000003, any_hit=False),
        # shadow rays against a mid-size resident scene
        dict(name="query_shadow", kind="trace", tris=130000, rays=262144, any_hit=True),
        # the smallest frame: the Cornell box from host buffers, re-uploaded and read back as the reference does
        dict(name="frame_cornell_host", kind="cornell", width=320, height=180, spp=16, depth=8),
        # an ordinary frame on the plain path (8 lanes per pixel, adaptive sampling) of a resident scene
        dict(name="frame_plain", kind="plain", tris=150000, width=1280, height=720, spp=16, depth=10),
        # a small odd-sized ReSTIR frame with the denoiser from host buffers
        dict(name="frame_restir_small_host", kind="restir_host", tris=20000, width=333, height=187, spp=4, depth=6),
        # the headline: ReSTIR and denoiser at 1280x720, 64 spp, depth 12, over 1,028,098 triangles
        dict(name="frame_restir_large", kind="restir", tris=1028098, width=1280, height=720, spp=64, depth=12),
        # one frame of an animation: deforming mesh uploaded, world rebuilt on the device, BVH refitted, frame rendered
        dict(name="frame_animated", kind="animated", spheres=200, cloth=256, width=1280, height=720, spp=16, depth=12),
        # a scene loaded (upload, checks, BVH build) and its first preview frame
        dict(name="scene_load", kind="load", tris=400000, width=160, height=90),
        # many uneven images in one call
        dict(name="batch_uneven", kind="batch", images=8, tris=60000, width=1280, height=720, spp=16, depth=10),
        # a step of a material fit: materials set, forward frame, gradient of an L2 loss
        dict(name="fit_step_plain", kind="fit", restir=False, spheres=100, ground=190, width=512, height=512, spp=32,
             depth=8),
        # the same on the ReSTIR chain with the denoiser
        dict(name="fit_step_restir", kind="fit", restir=True, spheres=40, ground=64, width=256, height=256, spp=16,
             depth=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame(rng, most):
    """An image of at most about `most` pixels, odd sizes among them."""
    px = _log(rng, 4000, most)
    aspect = rng.choice((1.0, 4 / 3, 16 / 9, 16 / 9, 21 / 9))
    h = max(16, int(round(math.sqrt(px / aspect))))
    return max(16, int(round(h * aspect))) + rng.randrange(4), h + rng.randrange(3)


def draw(rng):
    kind = rng.choice(("noalloc", "trace", "cornell", "plain", "restir_host", "restir", "animated", "load", "batch",
                       "fit", "trace", "restir"))
    if kind == "noalloc":
        return dict(kind=kind, tris=_log(rng, 100, 60000), rays=_log(rng, 256, 400000), any_hit=rng.random() < 0.4)
    if kind == "trace":
        return dict(kind=kind, tris=_log(rng, 2000, 512000), rays=_log(rng, 4096, 1000003), any_hit=rng.random() < 0.5)
    if kind == "cornell":
        w, h = _frame(rng, 320 * 180)
        return dict(kind=kind, width=w, height=h, spp=rng.choice((1, 4, 16, 32, 50)), depth=rng.randint(2, 8))
    if kind == "load":
        return dict(kind=kind, tris=_log(rng, 1000, 400000), width=rng.randint(64, 320), height=rng.randint(36, 180))
    if kind == "animated":
        w, h = _frame(rng, 1280 * 720)
        return dict(kind=kind, spheres=_log(rng, 20, 200), cloth=rng.randint(32, 256), width=w, height=h,
                    spp=rng.choice((1, 4, 8, 16)), depth=rng.randint(4, 12))
    if kind == "batch":
        w, h = _frame(rng, 1280 * 720)
        return dict(kind=kind, images=rng.randint(2, 8), tris=_log(rng, 2000, 60000), width=w, height=h,
                    spp=rng.choice((4, 8, 16)), depth=rng.randint(4, 12))
    if kind == "fit":
        restir = rng.random() < 0.5
        w, h = _frame(rng, 256 * 256 if restir else 512 * 512)
        return dict(kind=kind, restir=restir, spheres=_log(rng, 10, 100), ground=rng.randint(20, 190), width=w,
                    height=h, spp=rng.choice((2, 4, 8, 16) if restir else (2, 4, 8, 16, 32)), depth=rng.randint(3, 8))
    w, h = _frame(rng, 1280 * 720)
    if kind == "restir_host":
        return dict(kind=kind, tris=_log(rng, 2000, 100000), width=w, height=h, spp=rng.choice((1, 2, 4, 8)),
                    depth=rng.randint(2, 12))
    if kind == "plain":
        return dict(kind=kind, tris=_log(rng, 1000, 500000), width=w, height=h, spp=rng.choice((1, 4, 8, 16, 32, 64)),
                    depth=rng.randint(4, 12))
    return dict(kind="restir", tris=_log(rng, 5000, 500000), width=w, height=h, spp=rng.choice((1, 8, 16, 32, 64)),
                depth=rng.randint(4, 12))


# ---------------------------------------------------------------- inputs

def _field(seed, tris, width=64, height=36, spp=1, depth=4):
    """(SceneBuilder, Camera, RenderConfig) of an icosphere field of about `tris` triangles; the full-size one is
    icosphere_field's own."""
    if tris >= 1028098:
        return icosphere_field(seed, width=width, height=height, spp=spp, depth=depth)
    return sized_field(seed, tris, width, height, spp, depth)


def _restir(cfg):
    """The settings of the ReSTIR chain with the denoiser (32 candidates, 5 neighbours, radius 30 px)."""
    cfg.restir_candidates, cfg.restir_spatial, cfg.restir_radius = 32, 5, 30.0
    cfg.flags = _abi.RM_FLAG_NO_ENV
    return cfg


def _rays(seed, n):
    """Rays between random points of the field's volume: half of them start on a shared origin (a sensor), half
    anywhere."""
    rng = np.random.default_rng(seed + 77)
    o = rng.uniform([-22, 0.1, -22], [22, 12, 22], (n, 3))
    o[: n // 2] = o[0]
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.empty((n, 7), np.float32)
    rays[:, :3], rays[:, 3:6], rays[:, 6] = o, d, FAR
    return rays


class _Scene:
    """A scene object and the backend it lives on."""

    def __init__(self, backend, packed):
        self.backend, self.h = backend, backend.scene_create(packed)

    def __del__(self):
        if getattr(self.backend, "h", None):
            self.backend.scene_destroy(self.h)


def _images(npix):
    return (torch.empty(npix * 3, dtype=torch.uint8, device="cuda"),
            torch.empty(npix * 3, dtype=torch.float32, device="cuda"))


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case, seed=1000 + seed)
    scene_seed = seed % 100003
    if kind in ("noalloc", "trace"):
        packed = _field(scene_seed, case["tris"])[0].pack()
        st["rays"] = torch.from_numpy(_rays(seed, case["rays"])).cuda()
        st["tri"] = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
        st["tuv"] = [torch.empty(case["rays"], device="cuda") for _ in range(3)]
        if kind == "noalloc":
            st["lib"] = rb.load_library()
            st["tris"] = torch.from_numpy(packed.tris.view(np.uint8)).cuda()
            st["n_tris"] = packed.n_tris
            st["err"] = C.create_string_buffer(512)
            return st
    if kind == "animated":
        seq = AnimatedSequence(seed=scene_seed, n_spheres=case["spheres"], cloth_verts=case["cloth"],
                               width=case["width"], height=case["height"], spp=case["spp"], depth=case["depth"])
        st["b"] = b = rb.Backend(0)
        ids = np.asarray([b.model_create(m) for m in seq.models], np.int32)
        st["cloth_id"], st["cloth"] = int(ids[seq.CLOTH]), [seq.cloth(f) for f in range(3)]
        st["world"] = [objects.instance_records(seq.instances(f)) for f in range(3)]
        for r in st["world"]:
            r["model"] = ids[r["model"]]
        st["cams"], st["cfg"], st["frame"] = [seq.camera(f) for f in range(3)], seq.cfg, 0
        st["cfg"].flags |= _abi.RM_FLAG_NO_ENV
        st["rgb"], st["hdr"] = _images(case["width"] * case["height"])
        return st
    if kind == "batch":
        st["b"] = b = rb.Backend(0)
        rng = np.random.default_rng(scene_seed)
        st["scenes"], st["items"], st["out"] = [], [], []
        for k in range(case["images"]):
            # uneven: each image with its own scene, size and sample count up to the case's
            n = int(case["tris"] ** (1 - 0.4 * k / case["images"]))
            shrink = (1.0, 0.5, 0.7, 0.35)[k % 4]
            w, h = max(8, int(case["width"] * shrink)), max(8, int(case["height"] * shrink))
            spp = max(1, case["spp"] >> (k % 3))
            sb, cam, cfg = sized_field(scene_seed * 16 + k, n, w, h, spp, case["depth"])
            st["scenes"].append(_Scene(b, sb.pack()))
            rgb, hdr = _images(w * h)
            st["out"] += [rgb, hdr]
            st["items"].append(rb.BatchItem(st["scenes"][-1].h, cam, cfg, int(rng.integers(1 << 31)), rgb.data_ptr(),
                                            hdr.data_ptr()))
        return st
    if kind == "fit":
        d = inverse_scene(scene_seed, n_spheres=case["spheres"], n_dielectric=case["spheres"] // 3,
                          ground=case["ground"], width=case["width"], height=case["height"], spp=case["spp"],
                          depth=case["depth"])
        st["b"] = b = rb.Backend(0)
        st["stream"] = torch.cuda.Stream()
        b.set_stream(st["stream"].cuda_stream)
        st["cam"], st["cfg"] = d["camera"], d["config"]
        if case["restir"]:
            st["cfg"] = _restir(d["config"])
            st["cfg"].flags |= _abi.RM_FLAG_NOADAPT
        st["scene"] = _Scene(b, d["scene"])
        # the start of the fit: parameters off by up to 30 %, the light table of their emission
        rng = np.random.default_rng(scene_seed + 9)
        prm = np.where(d["mask"], d["params"] * rng.uniform(0.7, 1.3, d["params"].shape), d["params"])
        prm = prm.astype(np.float32)
        prm[:, 0:4] = np.clip(prm[:, 0:4], 0.05, 0.95)
        moved = with_materials(d["scene"], d["tri_material"], prm)
        st["params"], st["cdf"], st["total"] = prm, moved.light_cdf, moved.light_total
        b.scene_set_materials(st["scene"].h, prm, d["tri_material"], moved.light_cdf, moved.light_total)
        npix = case["width"] * case["height"]
        st["rgb"], st["hdr"] = _images(npix)
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["target"] = torch.rand(npix * 3, device="cuda", generator=g)
        st["dl"] = torch.empty_like(st["target"])
        st["grad"] = torch.zeros(len(prm) * 8, device="cuda")
        return st
    if kind == "cornell":
        sb, st["cam"], st["cfg"] = cornell_box(scene_seed)
        c = st["cfg"]
        c.width, c.height, c.spp, c.max_bounces = (case[k] for k in ("width", "height", "spp", "depth"))
        c.flags |= _abi.RM_FLAG_NO_ENV
        st["packed"] = sb.pack()
    elif kind == "load":
        sb, st["cam"], st["cfg"] = _field(scene_seed, case["tris"], case["width"], case["height"], 1, 4)
        st["packed"] = sb.pack()
    elif kind != "trace":
        sb, st["cam"], st["cfg"] = _field(scene_seed, case["tris"], case["width"], case["height"], case["spp"],
                                          case["depth"])
        if kind == "plain":
            st["cfg"].restir_candidates, st["cfg"].flags = 1, PLAIN_FLAGS
        else:
            _restir(st["cfg"])
        packed = sb.pack()
        if kind == "restir_host":
            st["packed"] = packed
    st["b"] = rb.Backend(0)
    if kind == "trace":
        st["b"].upload(packed, use_nodes=False)
    elif kind in ("plain", "restir"):
        st["b"].upload(packed, use_nodes=False)
        st["rgb"], st["hdr"] = _images(case["width"] * case["height"])
    elif kind == "load":
        st["rgb"], st["hdr"] = _images(case["width"] * case["height"])
    else:
        st["image"] = np.empty(case["width"] * case["height"] * 3, np.uint8)
    st["frame"] = 0
    return st


# ---------------------------------------------------------------- one pass

def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "noalloc":
        t, u, v = st["tuv"]
        rc = st["lib"].rmcuda_trace_noalloc(st["tris"].data_ptr(), st["n_tris"], st["rays"].data_ptr(), case["rays"],
                                            int(case["any_hit"]), st["tri"].data_ptr(), t.data_ptr(), u.data_ptr(),
                                            v.data_ptr(), torch.cuda.current_stream().cuda_stream, st["err"], 512)
        if rc != _abi.RM_OK:
            raise RuntimeError(st["err"].value.decode())
        return _hits(st)
    b = st["b"]
    if kind == "trace":
        t, u, v = st["tuv"]
        if case["any_hit"]:
            b.trace(st["rays"].data_ptr(), case["rays"], True, st["tri"].data_ptr())
        else:
            b.trace(st["rays"].data_ptr(), case["rays"], False, st["tri"].data_ptr(), t.data_ptr(), u.data_ptr(),
                    v.data_ptr())
        return _hits(st)
    if kind == "batch":
        b.render_batch(st["items"])
        return st["out"]
    if kind == "fit":
        h = st["scene"].h
        with torch.cuda.stream(st["stream"]):
            b.scene_set_materials(h, st["params"], None, st["cdf"], st["total"])
            b.render_scene_async(h, st["cam"], st["cfg"], st["seed"], st["rgb"].data_ptr(), st["hdr"].data_ptr())
            torch.sub(st["hdr"], st["target"], out=st["dl"])
            st["dl"].mul_(2.0 / st["dl"].numel())
            st["grad"].zero_()
            b.backward(h, st["cam"], st["cfg"], st["seed"], st["dl"].data_ptr(), st["grad"].data_ptr())
        return dict(rgb=st["rgb"], hdr=st["hdr"], grad=st["grad"])
    if kind == "load":
        h = b.scene_create(st["packed"])
        b.render_scene_async(h, st["cam"], st["cfg"], st["seed"], st["rgb"].data_ptr(), st["hdr"].data_ptr())
        b.scene_destroy(h)
        return dict(rgb=st["rgb"], hdr=st["hdr"])
    f = st["frame"]  # frames of one view follow one another with new seeds, as an animation's do
    st["frame"] += 1
    seed = st["seed"] + f
    if kind in ("cornell", "restir_host"):
        rgb, hdr = b.render(st["packed"], st["cam"], st["cfg"], seed, hdr=True, use_nodes=False, out=st["image"])
        return dict(rgb=rgb, hdr=hdr)
    cam = st["cam"] if kind != "animated" else st["cams"][f % 3]
    if kind == "animated":
        b.model_update(st["cloth_id"], st["cloth"][f % 3])
        b.instances_commit(st["world"][f % 3], rebuild_every=32)
    b.render_resident_async(cam, st["cfg"], seed, st["rgb"].data_ptr(), st["hdr"].data_ptr())
    return dict(rgb=st["rgb"], hdr=st["hdr"])


def _hits(st):
    """Closest hits whole; of an any-hit query the occlusion, which is all it promises (the triangle is some hit)."""
    if st["case"]["any_hit"]:
        return dict(occluded=st["tri"] >= 0)
    t, u, v = st["tuv"]
    return dict(tri=st["tri"], t=t, u=u, v=v)


# ---------------------------------------------------------------- work and 64-bit values

def work(case):
    """Bytes: the scene's triangles (176 each), rays, and images once.  Flops: one closest-hit ray per sample and its
    light sample: two boxes per level of a binary tree (24 flops a box) and one triangle (50 flops), 60 flops per light
    candidate, 150 for a surface sample; a fit step twice that.  Later vertices depend on the scene and are left
    out."""
    kind = case["kind"]
    tris = {"cornell": 36, "animated": case.get("spheres", 0) * 5120 + 4098 + 2 * (case.get("cloth", 1) - 1) ** 2,
            "fit": case.get("spheres", 0) * 1280 + 2 * case.get("ground", 0) ** 2 + 32}.get(kind, case.get("tris", 0))
    ray = math.log2(max(2, tris)) * 48 + 50
    if kind in ("noalloc", "trace"):
        n = case["rays"]
        return dict(bytes=tris * 176.0 + n * (28 + (4 if case["any_hit"] else 16)), flops=n * ray)
    px = case["width"] * case["height"]
    spp = case.get("spp", 1)
    if kind == "batch":
        px, tris = px * case["images"] * 0.45, tris * case["images"] * 0.5
        spp *= 0.6
    candidates = 32 if kind in ("restir", "restir_host", "animated") or case.get("restir") else 1
    flops = px * spp * (2 * ray + 60 * candidates + 150)
    return dict(bytes=tris * 176.0 + px * 15, flops=flops * (2 if kind == "fit" else 1))


def exact(case, seed):
    """Hits of a query by testing every triangle in 64 bits; the frames are random walks whose decisions no other
    precision repeats, so they have no such value."""
    if case["kind"] not in ("noalloc", "trace") or case["any_hit"]:
        return None
    packed = _field(seed % 100003, case["tris"])[0].pack()
    if packed.n_tris * case["rays"] > 4_000_000_000:
        return None
    rays = torch.from_numpy(_rays(seed, case["rays"])).cuda().double()
    v0, v1, v2 = (torch.from_numpy(np.ascontiguousarray(packed.tris[k])).cuda().double() for k in ("v0", "v1", "v2"))
    e1, e2 = v1 - v0, v2 - v0
    n = torch.linalg.cross(e1, e2)
    tri = torch.full((case["rays"],), -1, dtype=torch.int64, device="cuda")
    t, u, v = rays[:, 6].clone(), torch.zeros_like(rays[:, 6]), torch.zeros_like(rays[:, 6])
    step = max(1, 30_000_000 // packed.n_tris)
    for i in range(0, case["rays"], step):
        o, d = rays[i:i + step, :3], rays[i:i + step, 3:6]
        # Moeller-Trumbore with s = o - v0, as products of the ray's moment m = o x d and per-triangle terms:
        # det = -d.n, u = d.(e2 x s) / det, v = d.(s x e1) / det, t = s.n / det
        m = torch.linalg.cross(o, d)
        det = -(d @ n.T)
        c2 = torch.linalg.cross(v0, e2)
        c1 = torch.linalg.cross(v0, e1)
        uu = (m @ e2.T + d @ c2.T) / det
        vv = -(m @ e1.T + d @ c1.T) / det
        tt = (o @ n.T - (v0 * n).sum(1)) / det
        ok = (det.abs() >= 1e-12) & (uu >= 0) & (uu <= 1) & (vv >= 0) & (uu + vv <= 1) & (tt > 1e-8)
        ok &= tt < rays[i:i + step, 6:7]
        best, k = torch.where(ok, tt, math.inf).min(1)
        hit = torch.isfinite(best)
        row = torch.arange(len(k), device="cuda")
        tri[i:i + step] = torch.where(hit, k, -1)
        t[i:i + step] = torch.where(hit, best, t[i:i + step])
        u[i:i + step] = torch.where(hit, uu[row, k], 0.0)
        v[i:i + step] = torch.where(hit, vv[row, k], 0.0)
    return dict(tri=tri.int(), t=t, u=u, v=v)
