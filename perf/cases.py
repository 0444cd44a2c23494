"""Timing cases: what a program that uses this package has it do.

A case is a dict of plain values; listed() names the standing ones, draw()
gives further ones over the same ranges.  Kinds:

  frame    one progressive frame of an interactive viewer: Renderer.render_batch
           (sample_per_frame samples per pixel folded into the film), the
           accumulated film into a device buffer, tone mapping to 8 bits there
  still    render(scene, spp) -> HDR image in host memory
  guided   a chunk of samples rendered with an already trained guide
  train    a chunk of online training of a guide: its weights, its loss, the
           density it then has at a set of queries, and the chunk's image
  batch    render_batch over scenes of uneven size, resolution and budget
  rays     closest-hit and any-hit queries of a ray buffer, on host arrays or
           on device buffers
  build    the BVH built on the GPU (build_accel(builder="device"))

Scenes are the procedural ones of pathtracingtutorial_b200.scenes, seeded.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import pathtracingtutorial_b200 as pt
from pathtracingtutorial_b200 import scenes
from pathtracingtutorial_b200._ffi import check, lib

FLT_MAX = float(np.finfo(np.float32).max)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a preview window of the 36-triangle Cornell box;
        # launches and latency count
        dict(name="frame_cornell_256", kind="frame", scene="cornell", width=256, height=256, spf=4, depth=8),
        # the same viewer on a 2M-triangle field under an HDR sky at full HD
        dict(name="frame_field_1080p", kind="frame", scene="field", spheres=400, subdiv=4, width=1920, height=1080,
             spf=4, depth=16),
        # the small reference configuration: Cornell box, 512 x 512, 64 spp, depth 8, PCG
        dict(name="still_cornell_512", kind="still", scene="cornell", width=512, height=512, spp=64, depth=8),
        # every material texture path (alpha MASK and BLEND, normal maps, uv transforms), an odd size
        dict(name="still_textured", kind="still", scene="textured", width=803, height=601, spp=32, depth=8),
        # the headline workload: 2M triangles, full HD, 256 spp, depth 16, Sobol
        dict(name="still_field_1080p", kind="still", scene="field", spheres=400, subdiv=4, width=1920, height=1080,
             spp=256, depth=16),
        # hard indirect light: 200k-triangle closed room, long incoherent paths
        dict(name="still_room_1024", kind="still", scene="room", width=1024, height=1024, spp=64, depth=16),
        # the same room sampled with a trained guide (network inference every bounce)
        dict(name="guided_room_1024", kind="guided", scene="room", width=1024, height=1024, spp=32, depth=16,
             train_spp=8),
        # online training of the guide
        dict(name="train_room_512", kind="train", scene="room", width=512, height=512, spp=16, depth=16),
        # many scenes at once, uneven triangles, resolutions and budgets
        dict(name="batch_12_uneven", kind="batch", items=12, shape_seed=5, max_tris=200_000, max_spp=48, depth=12),
        # visibility queries of another program on this library's scene: a ray
        # buffer that lives on the device
        dict(name="rays_field_512k", kind="rays", scene="field", spheres=400, subdiv=3, rays=2_097_152, on_device=True),
        # the same queries from host arrays, few rays: the call's own cost
        dict(name="rays_cornell_20k", kind="rays", scene="cornell", rays=20_011, on_device=False),
        # geometry changed: the tree is rebuilt on the GPU
        dict(name="build_field_512k", kind="build", scene="field", spheres=400, subdiv=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "still", "still", "still", "guided", "train", "batch", "rays", "rays", "build"])
    c = dict(kind=kind)
    if kind in ("frame", "still"):
        c["scene"] = rng.choice(["cornell", "textured", "field", "room"])
    elif kind in ("guided", "train"):
        c["scene"] = "room"
    elif kind == "rays":
        c["scene"] = rng.choice(["cornell", "field", "room"])
    elif kind == "build":
        c["scene"] = rng.choice(["field", "room"])
    if c.get("scene") == "field":
        c["spheres"], c["subdiv"] = _log_int(rng, 12, 400), rng.choice([2, 3, 4])
    if kind in ("frame", "still", "guided", "train"):
        hi = 512 if kind == "train" else 1400
        c["width"], c["height"] = _log_int(rng, 192, hi), _log_int(rng, 192, min(hi, 1080))
        c["depth"] = rng.choice([8, 12, 16])
    if kind == "frame":
        c["spf"] = rng.choice([1, 2, 4, 8])
    elif kind == "still":
        c["spp"] = _log_int(rng, 8, 96)
    elif kind == "guided":
        c["spp"], c["train_spp"] = _log_int(rng, 4, 32), 8
    elif kind == "train":
        c["spp"] = _log_int(rng, 4, 16)
    elif kind == "batch":
        c["items"], c["shape_seed"] = rng.randint(2, 12), rng.randint(0, 9999)
        c["max_tris"], c["max_spp"], c["depth"] = _log_int(rng, 2_000, 200_000), rng.randint(8, 48), 12
    elif kind == "rays":
        c["rays"], c["on_device"] = _log_int(rng, 5_000, 2_000_000), rng.random() < 0.6
    if kind in ("frame", "still"):
        c["sampler"] = rng.choice(["pcg", "sobol"])
        if rng.random() < 0.25:
            c["watertight"] = True
        if rng.random() < 0.25:
            c["aperture"] = 0.02
    return c


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _arrays(case, seed):
    kind = case["scene"]
    size = dict(width=case.get("width", 64), height=case.get("height", 64), spp=case.get("spp", case.get("spf", 4)),
                max_depth=case.get("depth", 8))
    if kind == "field":
        sa = scenes.icosphere_field(n_spheres=case["spheres"], subdiv=case["subdiv"], seed=seed,
                                    env_size=(2048, 1024) if "width" in case else None, **size)
    elif kind == "room":
        sa = scenes.hidden_light_room(seed=seed, **size)
    else:
        make = scenes.cornell_box if kind == "cornell" else scenes.textured_cornell
        sa = make(pcg_seed=1 + seed % 1_000_000, **size)
        # another seed is another room: wall colours and the viewpoint move
        rng = np.random.default_rng(seed)
        sa.materials["base_color"] *= rng.uniform(0.8, 1.0, (len(sa.materials), 3)).astype(np.float32)
        sa.camera["position"] += rng.uniform(-0.05, 0.05, 3).astype(np.float32)
    if "sampler" in case:
        sa.sampler = {"pcg": pt.SAMPLER_PCG, "sobol": pt.SAMPLER_SOBOL}[case["sampler"]]
        sa.pcg_seed = 1 + seed % 1_000_000
    if "spf" in case:
        sa.sample_per_frame = case["spf"]
    if "aperture" in case:
        sa.camera["aperture"] = case["aperture"]
        sa.camera["focal_distance"] = float(np.linalg.norm(sa.camera["position"] - sa.camera["look_at"]))
    return sa


def _scene(case, seed):
    sa = _arrays(case, seed)
    s = sa.scene()
    if case.get("watertight"):
        s.update_settings(flags=pt.FLAG_WATERTIGHT)
    s.build_accel()
    s.upload_to_device(0)
    return sa, s


def _batch_shapes(case):
    """(spheres, subdiv, width, height, spp) per item: fixed by the case, as the
    items' sizes are a property of the job."""
    rng = np.random.default_rng(case["shape_seed"])
    out = []
    for _ in range(case["items"]):
        target = float(np.exp(rng.uniform(np.log(1_000), np.log(case["max_tris"]))))
        sub = next(s for s in (1, 2, 3, 4) if target / (20 * 4 ** s) <= 400 or s == 4)
        w, h = [(256, 256), (512, 512), (1024, 1024), (1280, 720)][int(rng.integers(0, 4))]
        out.append((max(1, int(round(target / (20 * 4 ** sub)))), sub, w, h, int(rng.integers(4, case["max_spp"] + 1))))
    return out


def _rays(case, seed, sa):
    """Origins spread through the space above the scene's floor, directions
    uniform on the sphere, occlusion distances up to the scene's extent."""
    rng = np.random.default_rng(seed + 1)
    p = sa.vertices["position"]
    if case["scene"] == "field":
        lo, hi = np.float32([-22, 0.01, -22]), np.float32([22, 4.0, 13])
    else:
        lo, hi = p.min(0), p.max(0)
    n = case["rays"]
    o = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tmax = rng.uniform(0.1, 1.0, n).astype(np.float32) * np.float32((hi - lo).max())
    return o, d, tmax


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "batch":
        env = scenes.sky_env(1024, 512)
        st["items"] = []
        for k, (n, sub, w, h, spp) in enumerate(_batch_shapes(case)):
            sa = scenes.icosphere_field(n_spheres=n, subdiv=sub, width=w, height=h, spp=spp, max_depth=case["depth"],
                                        seed=seed + 1000 * k, env_size=None)
            sa.env = env
            s = sa.scene()
            s.build_accel()
            s.upload_to_device(0)
            st["items"].append((s, spp))
        return st
    if kind == "build":
        sa = _arrays(case, seed)
        st["scene"] = sa.scene()
        # room for the tree: fewer inner nodes than triangles, one record per triangle
        st["inner"] = np.zeros((len(sa.faces), 16), np.int32)
        st["tris"] = np.zeros((len(sa.faces), 12), np.int32)
        return st
    sa, s = _scene(case, seed)
    st["scene"] = s
    if kind == "rays":
        o, d, tmax = _rays(case, seed, sa)
        if case["on_device"]:
            st["rays"] = torch.from_numpy(pt._pack_rays(o, d, tmax)).cuda()
            st["hits"] = torch.empty((len(o), 4), dtype=torch.int32, device="cuda")
            st["occ"] = torch.empty(len(o), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
        else:
            st["rays"] = (o, d, tmax)
    elif kind == "frame":
        st["renderer"] = pt.Renderer(s)
        st["rgba"] = torch.zeros((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        st["rgba8"] = torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
    elif kind in ("guided", "train"):
        r = st["renderer"] = pt.Renderer(s)
        g = st["guide"] = pt.Guide(s, seed=1 + seed % 1_000_000)
        spf = s.settings().sample_per_frame
        st["frames"] = max(1, case["spp"] // spf)
        g.attach(r.integrator, pt.Guide.TRAIN)
        if kind == "guided":
            s.set_frame_count(100_000)
            r.render_frames(case["train_spp"] // spf)
            g.attach(r.integrator, pt.Guide.USE)
            r.reset_accumulation()
        else:
            rng = np.random.default_rng(seed + 2)
            p = sa.vertices["position"]
            st["pos"] = rng.uniform(p.min(0), p.max(0), (4096, 3)).astype(np.float32)
            st["dir"] = rng.normal(size=(4096, 3)).astype(np.float32)
        r.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "still":
        return pt.render(st["scene"], case["spp"])
    if kind == "frame":
        r = st["renderer"]
        r.render_batch()
        check(lib().pt_film_download_to(r.film._h, C.c_void_p(st["rgba"].data_ptr()), 1))
        check(lib().pt_tonemap(C.c_void_p(st["rgba"].data_ptr()), case["width"], case["height"], -2.8,
                               C.c_void_p(st["rgba8"].data_ptr()), 1, 0))
        return {"film": st["rgba"], "display": st["rgba8"]}
    if kind == "guided":
        r = st["renderer"]
        r.render_frames(st["frames"])
        return r.download_current_image()
    if kind == "train":
        r, g = st["renderer"], st["guide"]
        r.render_frames(st["frames"])
        return {"weights": g.params(with_grid=False)["weights"], "loss": g.loss(), "pdf": g.pdf(st["pos"], st["dir"]),
                "image": r.download_current_image()}
    if kind == "batch":
        return pt.render_batch(st["items"], autotune=False, mode=pt.BATCH_WAVEFRONT)[0]
    if kind == "rays":
        if case["on_device"]:
            s, n, rays = st["scene"].handle, len(st["rays"]), C.c_void_p(st["rays"].data_ptr())
            check(lib().pt_trace_closest(s, rays, n, C.c_void_p(st["hits"].data_ptr()), 1))
            check(lib().pt_trace_any(s, rays, n, C.c_void_p(st["occ"].data_ptr()), 1))
            return {"t": st["hits"][:, 0].view(torch.float32), "prim": st["hits"][:, 1],
                    "uv": st["hits"][:, 2:].view(torch.float32), "occluded": st["occ"]}
        o, d, tmax = st["rays"]
        h = pt.trace_closest(st["scene"], o, d)
        return {"t": h["t"], "prim": h["prim"], "uv": np.stack([h["u"], h["v"]], 1),
                "occluded": pt.trace_any(st["scene"], o, d, tmax)}
    s = st["scene"]
    s.build_accel(builder="device")
    inner, tris, root = st["inner"], st["tris"], C.c_uint32(0)
    check(lib().pt_scene_get_traversal(s.handle, pt._ffi.ptr(inner), len(inner), pt._ffi.ptr(tris), len(tris),
                                       C.byref(root)))
    return {"inner": inner, "tris": tris, "root": int(root.value)}


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------
def _triangles(case):
    return {"cornell": 36, "textured": 40, "room": 202_002}.get(case["scene"]) or \
        case["spheres"] * 20 * 4 ** case["subdiv"] + 2


def _path_flops(tris, depth, env):
    """Arithmetic of one path: per ray a descent of about log2(tris) nodes (two
    box tests of 24 operations each) and four triangle tests of 50; two rays
    per vertex (the next one and the light's) and about 600 operations of
    shading.  Open scenes lose most paths to the sky after two vertices, closed
    ones run to the roulette."""
    vertices = min(depth, 2.0 if env else 5.0)
    ray = 48.0 * max(1.0, math.log2(tris)) + 200.0
    return vertices * (2.0 * ray + 600.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        by, fl = 8.0 * 1024 * 512, 0.0
        for n, sub, w, h, spp in _batch_shapes(case):
            tris = n * 20 * 4 ** sub + 2
            by += 110.0 * tris + 16.0 * w * h
            fl += w * h * spp * _path_flops(tris, case["depth"], True)
        return {"bytes": by, "flops": fl}
    tris = _triangles(case)
    geometry = 112.0 * tris                  # triangle records and nodes, each once
    if kind == "rays":
        ray = 48.0 * max(1.0, math.log2(tris)) + 200.0
        return {"bytes": geometry + case["rays"] * (32.0 + 16.0 + 32.0 + 1.0), "flops": 2.0 * case["rays"] * ray}
    if kind == "build":
        # vertices (about half as many as triangles) and faces in; nodes, triangle records and faces out
        return {"bytes": tris * (32.0 + 16.0 + 64.0 + 48.0 + 16.0), "flops": 0.0}
    pixels = case["width"] * case["height"]
    env = case["scene"] == "field"
    paths = pixels * case.get("spf" if kind == "frame" else "spp")
    by = geometry + (16.0 * 2048 * 1024 if env else 0.0) + 16.0 * pixels + (36.0 * pixels if kind == "frame" else 0.0)
    fl = paths * _path_flops(tris, case["depth"], env)
    if kind in ("guided", "train"):
        by += 16 * 2 ** 19 * 4.0
        fl += paths * 5.0 * 26_000.0 * (4.0 if kind == "train" else 1.0)   # the network, once per vertex
    return {"bytes": by, "flops": fl}


def exact(case, seed):
    """Closest hits and occlusion of the ray queries by brute force over all
    triangles in 64 bits, where that is quick.  A rendered image has no such
    value: its paths branch on 32-bit comparisons."""
    if case["kind"] != "rays" or case["scene"] != "cornell" or case["rays"] > 200_000:
        return None
    sa = _arrays(case, seed)
    o, d, tmax = (a.astype(np.float64) for a in _rays(case, seed, sa))
    p = sa.vertices["position"].astype(np.float64)
    n = len(o)
    t, uv = np.full(n, FLT_MAX), np.zeros((n, 2))
    for f in sa.faces:
        v0, v1, v2 = p[f["v0"]], p[f["v1"]], p[f["v2"]]
        e1, e2 = v1 - v0, v2 - v0
        q = np.cross(d, e2)
        det = q @ e1
        with np.errstate(divide="ignore", invalid="ignore"):
            inv = 1.0 / det
            s = o - v0
            u = np.einsum("ij,ij->i", s, q) * inv
            r = np.cross(s, e1)
            v = np.einsum("ij,ij->i", d, r) * inv
            tt = (r @ e2) * inv
            ok = (np.abs(det) > 1e-7) & (u >= 0) & (v >= 0) & (u + v <= 1) & (tt >= 1e-4) & (tt < t)
        t = np.where(ok, tt, t)
        uv = np.where(ok[:, None], np.stack([u, v], 1), uv)
    # triangle numbers and the occlusion flags are whole values
    return {"t": t, "prim": None, "uv": uv, "occluded": None}
