"""Performance cases of the GB300 path tracer.

Each case is work that a program using the library has it do, through the
public binding (cpppt.lib): ray batches in device and in host memory, renders
from one-sample previews to full frames, multi-scene batches, renders with
the learned guide (frozen and training) and with the SD-tree, and the
creation of a scene.  Scenes, resolutions, sample counts and depths are those
of the repository's own workloads: the Cornell box (256x256, depth 8), the
triangle soup of geodesic spheres (2000 spheres = 1M triangles, 1920x1080,
depth 10), the room with the light behind a slit (1000 boxes = 192k
triangles, 1280x720, depth 12) and the batch of eight small soups.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpp-pt_gb300"))

from cpppt import scenes  # noqa: E402
from cpppt.lib import (FLAG_NN_FREEZE, FLAG_UNBIASED_MIS, MODE_MIS, MODE_NEE, MODE_NN, MODE_PT,  # noqa: E402
                       MODE_SDTREE, GpuBatch, GpuScene)

MODES = {"mis": (MODE_MIS, 0), "nee": (MODE_NEE, 0), "pt": (MODE_PT, 0), "unbiased": (MODE_MIS, FLAG_UNBIASED_MIS),
         "guided": (MODE_NN, FLAG_NN_FREEZE), "train": (MODE_NN, 0), "sdtree": (MODE_SDTREE, 0)}
DEPTH = {"cornell": 8, "soup": 10, "slit": 12}


def listed():
    return [
        # a program that asks for a few rays (picking, a visibility probe): latency
        {"name": "rays_1000", "call": "closest", "scene": "soup", "size": 40, "rays": 1000},
        # closest hits of a full frame's camera and bounce rays, an odd number of them
        {"name": "rays_frame", "call": "closest", "scene": "soup", "size": 2000, "rays": 1843201},
        # occlusion of as many shadow rays from surfaces toward the emitters
        {"name": "shadow_frame", "call": "any", "scene": "soup", "size": 2000, "rays": 1843199},
        # a ray batch in host memory, the drop-in for BVH::intersect on an array
        {"name": "rays_host", "call": "closest_host", "scene": "slit", "size": 250, "rays": 100003},
        # interactive preview: one sample per pixel of the large scene at a small resolution
        {"name": "preview_360p", "call": "render", "scene": "soup", "size": 2000, "width": 640, "height": 360, "spp": 1,
         "mode": "mis"},
        # the Cornell box as the reference renders it, image in host memory
        {"name": "cornell_64spp", "call": "render_host", "scene": "cornell", "size": 0, "width": 256, "height": 256,
         "spp": 64, "mode": "mis"},
        # the benchmark's frame
        {"name": "soup_1080p", "call": "render", "scene": "soup", "size": 2000, "width": 1920, "height": 1080, "spp": 16,
         "mode": "mis"},
        # eight uneven scenes in one wavefront
        {"name": "batch_8", "call": "batch", "scene": "soup", "size": 20, "width": 256, "height": 256, "spp": 4,
         "mode": "mis"},
        # the occluded-light room with a trained guide held fixed
        {"name": "guided_720p", "call": "render", "scene": "slit", "size": 1000, "width": 1280, "height": 720, "spp": 4,
         "mode": "guided"},
        # the same room with the guide learning while it renders
        {"name": "train_360p", "call": "train", "scene": "slit", "size": 1000, "width": 640, "height": 360, "spp": 8,
         "mode": "train"},
        # the reference's own guide
        {"name": "sdtree_cornell", "call": "render", "scene": "cornell", "size": 0, "width": 128, "height": 128,
         "spp": 64, "mode": "sdtree"},
        # loading geometry: both trees built on the device, and a first small query
        {"name": "scene_192k", "call": "create", "scene": "slit", "size": 1000, "rays": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["closest", "any", "closest_host", "any_host", "render", "render_host", "batch", "guided", "train",
                       "create"])
    scene = rng.choice(["soup", "slit"] if call != "render_host" else ["soup", "slit", "cornell"])
    size = {"soup": _log_int(rng, 20, 2000), "slit": _log_int(rng, 50, 1000), "cornell": 0}[scene]
    if call in ("closest", "any"):
        return {"call": call, "scene": scene, "size": size, "rays": _log_int(rng, 300, 1 << 21)}
    if call in ("closest_host", "any_host"):
        return {"call": call, "scene": scene, "size": size, "rays": _log_int(rng, 300, 300000)}
    if call == "create":
        return {"call": call, "scene": scene, "size": size, "rays": _log_int(rng, 256, 4096)}
    if call == "batch":
        s = rng.randrange(96, 321)
        return {"call": call, "scene": "soup", "size": _log_int(rng, 10, 60), "width": s, "height": s,
                "spp": rng.randrange(1, 9), "mode": rng.choice(["mis", "nee", "unbiased"])}
    width = _log_int(rng, 160, 1280)
    height = max(90, int(width * rng.uniform(0.5, 0.8)))
    if call == "train":  # one round of the wavefront (about 2^20 paths in flight), then the Adam steps on its records
        width, height = min(width, 1024), min(height, 720)
        return {"call": call, "scene": "slit", "size": size if scene == "slit" else 300, "width": width,
                "height": height, "spp": max(1, min(8, 1_600_000 // (width * height))), "mode": "train"}
    spp = max(1, min(_log_int(rng, 1, 64), 12_000_000 // (width * height)))
    if call == "guided":
        return {"call": "render", "scene": "slit", "size": size if scene == "slit" else 300, "width": width,
                "height": height, "spp": max(1, min(spp, 4_000_000 // (width * height))), "mode": "guided"}
    return {"call": call, "scene": scene, "size": size, "width": width, "height": height, "spp": spp,
            "mode": rng.choice(["mis", "mis", "nee", "pt", "unbiased"])}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _scene(case, seed):
    w, h = case.get("width", 1280), case.get("height", 720)
    if case["scene"] == "cornell":
        return scenes.cornell(w, h)
    if case["scene"] == "slit":
        return scenes.slit_room(seed=seed, n_boxes=case["size"], box_subdiv=4, width=w, height=h)
    return scenes.soup(seed=seed, n_spheres=case["size"], width=w, height=h)


def _camera_rays(sc, n, gen):
    """n camera rays of the scene, in scanline order of a frame of its aspect ratio, jittered."""
    cam = torch.tensor(np.asarray(sc.camera, np.float64), device="cuda")
    fwd = cam[3:6] - cam[0:3]
    fwd = fwd / fwd.norm()
    x = torch.linalg.cross(cam[6:9], -fwd)
    x = x / x.norm()
    y = torch.linalg.cross(-fwd, x)
    aspect = sc.width / sc.height
    cols = max(1, int(math.sqrt(n * aspect)))
    rows = -(-n // cols)
    k = torch.arange(n, device="cuda")
    jit = torch.rand(n, 2, device="cuda", generator=gen, dtype=torch.float64)
    u = (((k % cols) + jit[:, 0]) / cols) * 2 - 1
    v = 1 - ((k // cols + jit[:, 1]) / rows) * 2
    d = (u * cam[9] * aspect)[:, None] * x + (v * cam[9])[:, None] * y + fwd
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty(n, 7, device="cuda", dtype=torch.float32)
    rays[:, 0:3] = cam[0:3].float()
    rays[:, 3:6] = d.float()
    rays[:, 6] = math.inf
    return rays


def _directions(n, gen):
    d = torch.randn(n, 3, device="cuda", generator=gen)
    return d / d.norm(dim=1, keepdim=True)


def _surface_points(gs, sc, rays):
    """Points just off the surfaces that the rays hit, on the rays' side."""
    hits = torch.empty(len(rays), 4, device="cuda", dtype=torch.float32)
    gs.trace_closest_device(rays.data_ptr(), len(rays), hits.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    t = hits[:, 0:1]
    t = torch.where(torch.isfinite(t), t, torch.ones_like(t))
    return rays[:, 0:3] + rays[:, 3:6] * (t * 0.999)


def _closest_rays(gs, sc, n, gen):
    """Half camera rays, half bounce rays from the points that camera rays hit."""
    half = n // 2
    cam = _camera_rays(sc, n - half, gen)
    if half == 0:
        return cam
    rays = torch.empty(half, 7, device="cuda", dtype=torch.float32)
    rays[:, 0:3] = _surface_points(gs, sc, cam)[:half]
    rays[:, 3:6] = _directions(half, gen)
    rays[:, 6] = math.inf
    return torch.cat([cam, rays]).contiguous()


def _shadow_rays(gs, sc, n, gen):
    """Rays from the points that camera rays hit toward points on the emitters, ending just before them."""
    p = _surface_points(gs, sc, _camera_rays(sc, n, gen))
    emit = np.nonzero(np.asarray(sc.mat_kind)[sc.tri_material] == scenes.EMISSIVE)[0]
    tri = torch.tensor(np.asarray(sc.vertices)[np.asarray(sc.triangles)[emit]], device="cuda", dtype=torch.float32)
    pick = torch.randint(0, len(emit), (n,), device="cuda", generator=gen)
    b = torch.rand(n, 2, device="cuda", generator=gen)
    b = torch.where(b.sum(1, keepdim=True) > 1, 1 - b, b)
    q = tri[pick]
    target = q[:, 0] * (1 - b.sum(1, keepdim=True)) + q[:, 1] * b[:, 0:1] + q[:, 2] * b[:, 1:2]
    d = target - p
    dist = d.norm(dim=1, keepdim=True).clamp_min(1e-3)
    return torch.cat([p, d / dist, dist - 2e-4], dim=1).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    call = case["call"]
    st = {"case": case, "seed": seed % 100003}
    if call == "batch":
        w, h, n = case["width"], case["height"], case["size"]
        members = []
        for k in range(8):  # uneven triangle counts and resolutions
            m = 1 << (k % 3)
            members.append(GpuScene(scenes.soup(seed=seed + 31 * k, n_spheres=n << (k % 5), width=w * m, height=h * m)))
        st["gpu"] = GpuBatch(members)
        st["jobs"] = [dict(scene=k, spp=case["spp"], max_depth=10, seed=st["seed"] + k) for k in range(8)]
        st["out"] = [torch.zeros(s.height, s.width, 3, device="cuda") for s in members]
        return st
    sc = _scene(case, seed)
    gs = GpuScene(sc)
    if call == "create":
        st["scene"] = sc
        st["rays"] = _closest_rays(gs, sc, case["rays"], gen).cpu().numpy()
        gs.close()
        return st
    st["gpu"] = gs
    if call in ("closest", "any", "closest_host", "any_host"):
        n = case["rays"]
        any_hit = call.startswith("any")
        st["rays"] = (_shadow_rays if any_hit else _closest_rays)(gs, sc, n, gen)
        if call.endswith("host"):
            st["rays"] = st["rays"].cpu().numpy()
        else:
            st["out"] = torch.zeros(n, device="cuda", dtype=torch.uint8) if any_hit else torch.zeros(n, 4, device="cuda")
        torch.cuda.synchronize()
        return st
    st["out"] = torch.zeros(sc.height, sc.width, 3, device="cuda") if call != "render_host" else \
        np.zeros((sc.height, sc.width, 3), np.float32)
    if case["mode"] == "guided":  # a guide with the weights of a trained network's size
        gs.nn_reset(seed % 9973)
        gs.nn_set_weights(gs.nn_weights() * np.float32(1.5))
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    case, gs = st["case"], st.get("gpu")
    call = case["call"]
    if call == "closest":
        out = st["out"]
        gs.trace_closest_device(st["rays"].data_ptr(), len(st["rays"]), out.data_ptr(),
                                torch.cuda.current_stream().cuda_stream)
        return {"t": out[:, 0], "prim": out.view(torch.int32)[:, 1], "beta": out[:, 2], "gamma": out[:, 3]}
    if call == "any":
        gs.trace_any_device(st["rays"].data_ptr(), len(st["rays"]), st["out"].data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
        return {"occluded": st["out"]}
    if call == "closest_host":
        prim, t, beta, gamma = gs.trace_closest(st["rays"])
        return {"t": t, "prim": prim, "beta": beta, "gamma": gamma}
    if call == "any_host":
        return {"occluded": gs.trace_any(st["rays"])}
    if call == "create":
        g = GpuScene(st["scene"])
        prim, t, beta, gamma = g.trace_closest(st["rays"])
        g.close()
        return {"t": t, "prim": prim, "beta": beta, "gamma": gamma}
    mode, flags = MODES[case["mode"]]
    if call == "batch":
        gs.render_device(st["jobs"], [o.data_ptr() for o in st["out"]], mode=mode, flags=flags)
        return {"images": st["out"]}
    kw = dict(spp=case["spp"], max_depth=DEPTH[case["scene"]], seed=st["seed"], mode=mode, flags=flags)
    if call == "render_host":
        return {"image": gs.render(out=st["out"], **kw)}
    if call == "train":  # a guide learned from scratch for this frame
        gs.nn_reset(st["seed"])
        gs.render_device(st["out"].data_ptr(), **kw)
        return {"image": st["out"], "weights": gs.nn_weights()}
    gs.render_device(st["out"].data_ptr(), **kw)
    return {"image": st["out"]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _triangles(case, size=None):
    n = case["size"] if size is None else size
    return {"cornell": 36, "soup": 500 * n + 20, "slit": 192 * n + 38}[case["scene"]]


def _ray_work(tris):
    """Bytes and operations of one ray that descends straight to its triangle in
    a 4-wide tree: 64 B and 4 slab tests (12 operations each) per level, one
    triangle of 48 B (about 60 operations)."""
    levels = max(1, math.ceil(math.log(max(tris, 4) / 2, 4)))
    return 64 * levels + 48, 48 * levels + 60


def work(case):
    call = case["call"]
    if call == "batch":
        px = [case["width"] * case["height"] << (2 * (k % 3)) for k in range(8)]
        tris = [_triangles(case, case["size"] << (k % 5)) for k in range(8)]
        flops = sum(4 * p * case["spp"] * _ray_work(t)[1] for p, t in zip(px, tris))
        return {"bytes": 12 * sum(px) + 75 * sum(tris), "flops": flops}
    tris = _triangles(case)
    ray_bytes, ray_flops = _ray_work(tris)
    scene_bytes = 75 * tris  # 48 B per triangle and its share of the tree
    if call in ("closest", "closest_host", "any", "any_host"):
        n = case["rays"]
        io = n * (28 + (1 if call.startswith("any") else 16))
        return {"bytes": io + min(scene_bytes, n * ray_bytes), "flops": n * ray_flops}
    if call == "create":  # vertices and indices in, tree and triangles out, one pass per level of a binary tree
        return {"bytes": tris * (36 + 16 + 75), "flops": tris * 12 * math.ceil(math.log2(tris))}
    paths = case["width"] * case["height"] * case["spp"]
    flops = paths * 4 * ray_flops  # about four rays per path (extension and shadow)
    if case["mode"] in ("guided", "train"):  # inference at about three vertices per path
        flops += paths * 3 * 30720 * (3 if case["mode"] == "train" else 1)
    return {"bytes": 12 * case["width"] * case["height"] + scene_bytes, "flops": flops}


# ---------------------------------------------------------------------------
# Closest hits in 64 bits, every ray against every triangle
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["call"] not in ("closest", "closest_host", "create"):
        return None  # bytes, or Monte Carlo estimates of this library's own random numbers
    if case["rays"] * _triangles(case) > 2_000_000_000:
        return None
    st = prepare(case, seed)
    rays = torch.as_tensor(st["rays"], device="cuda").double()
    sc = st.get("scene") or _scene(case, seed)
    v = torch.tensor(np.asarray(sc.vertices)[np.asarray(sc.triangles)], device="cuda", dtype=torch.float64)
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = torch.linalg.cross(e1, e2)
    out = torch.empty(len(rays), 3, device="cuda", dtype=torch.float64)
    step = max(1, 40_000_000 // len(a))
    an, g1, g2 = (a * n).sum(1), torch.linalg.cross(e2, n), torch.linalg.cross(n, e1)
    nn = (n * n).sum(1)
    for k in range(0, len(rays), step):
        o, d = rays[k:k + step, 0:3], rays[k:k + step, 3:6]
        t = (an[None] - o @ n.T) / (d @ n.T)
        # barycentrics of the plane point o + t d: beta along e1, gamma along e2
        beta = ((o @ g1.T) + t * (d @ g1.T) - (a * g1).sum(1)[None]) / nn[None]
        gamma = ((o @ g2.T) + t * (d @ g2.T) - (a * g2).sum(1)[None]) / nn[None]
        ok = (t >= 1e-4) & (beta >= 0) & (gamma >= 0) & (beta + gamma <= 1)
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, j = t.min(dim=1)
        hit = torch.isfinite(best)
        out[k:k + step, 0] = best
        out[k:k + step, 1] = torch.where(hit, beta.gather(1, j[:, None])[:, 0], 0.0)
        out[k:k + step, 2] = torch.where(hit, gamma.gather(1, j[:, None])[:, 0], 0.0)
    return {"t": out[:, 0], "prim": None, "beta": out[:, 1], "gamma": out[:, 2]}
