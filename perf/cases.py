"""Performance cases of the Nova path tracer on one GPU, each a call (or the few calls) that a program
using the library makes, through its public entry points (axomae_b200.native over the C ABI).

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the program holds before the call: scene, contexts, buffers on the GPU
  run(state)           one pass; returns its outputs
  work(case)           bytes and operations one pass cannot do without
  exact(case, seed)    the outputs in 64 bits where they have such a value

Scenes are the repository's seeded generators (axomae_b200.scenes) with their own materials and
environment maps; the seed picks the scene, the inputs' values and the sampler's seed.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from axomae_b200 import native, scenes

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # an interactive preview: one sample per pixel of a small window, where launches and
        # latency count (the 64-sphere scene at a quarter of its default size)
        {"name": "preview_256", "kind": "frame", "scene": "spheres", "tris": 65536, "w": 256, "h": 256, "spp": 1,
         "depth": 4, "rr": -1, "bvh": 2},
        # one progressive frame of an editor viewport of ragged size: one sample per pixel, mixed
        # diffuse / conductor / dielectric materials
        {"name": "viewport_1283x721", "kind": "frame", "scene": "mixed", "tris": 150000, "w": 1283, "h": 721, "spp": 1,
         "depth": 8, "rr": -1, "bvh": 2},
        # a final frame at 1080p: a displaced ground of half a million triangles, several samples
        # per pixel (more paths than one wave holds), Russian roulette
        {"name": "final_1080p", "kind": "frame", "scene": "heightfield", "tris": 524288, "w": 1920, "h": 1080,
         "spp": 16, "depth": 8, "rr": 3, "bvh": 2},
        # an instanced scene with the two-level acceleration structure: rigid instances of a few meshes
        {"name": "instanced_720p", "kind": "frame", "scene": "instanced", "tris": 2000000, "w": 1280, "h": 720,
         "spp": 4, "depth": 6, "rr": -1, "bvh": 1},
        # a render farm's batch: frames of different scenes, sizes, sample counts and depths, scenes
        # already resident, films left on the device
        {"name": "batch_8", "kind": "batch", "jobs": 8, "tris": 300000, "side": 1024, "spp": 64, "depth": 12},
        # the same end to end: scenes from pinned host memory, builds, renders, films back in host memory
        {"name": "pipeline_4", "kind": "pipeline", "jobs": 4, "tris": 100000, "side": 384, "spp": 4, "depth": 6},
        # one step of inverse rendering: forward with per-triangle albedo and per-material roughness,
        # then the gradients of a per-pixel loss (the 64-sphere scene)
        {"name": "adjoint_256", "kind": "adjoint", "tris": 65536, "w": 256, "h": 256, "spp": 16, "depth": 4},
        # after an edit of the scene: upload, acceleration structure, the depth and normal images of the
        # viewport
        {"name": "scene_edit", "kind": "edit", "scene": "mixed", "tris": 150000, "w": 961, "h": 541, "bvh": 2},
        # the intersector by itself: closest hits of incoherent rays (picking, visibility, baking tools)
        {"name": "trace_1m", "kind": "trace", "tris": 65536, "n": 1000003},
        # the irradiance map of an environment, for image-based lighting
        {"name": "irradiance_512", "kind": "bake", "ow": 512, "oh": 256, "samples": 128, "sw": 2048, "sh": 1024,
         "ch": 4},
        # the bake command: .hdr file in, irradiance .hdr file out (decode, bake, encode)
        {"name": "bake_command", "kind": "command", "ow": 256, "oh": 128, "samples": 128, "sw": 1024, "sh": 512},
        # what follows every frame of a progressive 4K render: running mean, display image, snapshot
        {"name": "film_4k", "kind": "film", "w": 3840, "h": 2160, "ch": 4, "dw": 1920, "dh": 1080},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "pipeline", "adjoint", "edit", "trace", "bake", "command",
                       "film"])
    if kind == "frame":
        scene = rng.choice(["spheres", "mixed", "heightfield", "instanced"])
        w = _log(rng, 200, 1920)
        h = max(96, min(1080, int(w * rng.uniform(0.5, 1.0))))
        # between one frame of one sample and the largest listed one
        most = max(1, min(16, 33000000 // (w * h)))
        tris = {"spheres": (16384, 131072), "mixed": (20000, 300000), "heightfield": (32768, 524288),
                "instanced": (200000, 2000000)}[scene]
        return {"kind": kind, "scene": scene, "tris": _log(rng, *tris), "w": w, "h": h, "spp": rng.randint(1, most),
                "depth": rng.randint(2, 10), "rr": rng.choice([-1, 2, 3]),
                "bvh": rng.choice([1, 2]) if scene == "instanced" else 2}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 8), "tris": _log(rng, 20000, 300000), "side": _log(rng, 128, 1024),
                "spp": rng.choice([1, 4, 16, 64]), "depth": rng.choice([3, 6, 12])}
    if kind == "pipeline":
        return {"kind": kind, "jobs": rng.randint(2, 4), "tris": _log(rng, 20000, 100000), "side": _log(rng, 128, 384),
                "spp": rng.choice([1, 4]), "depth": rng.choice([3, 6])}
    if kind == "adjoint":
        w = _log(rng, 64, 320)
        return {"kind": kind, "tris": _log(rng, 16384, 131072), "w": w, "h": w - rng.randint(0, 31),
                "spp": rng.randint(1, 16), "depth": rng.randint(2, 6)}
    if kind == "edit":
        w = _log(rng, 320, 1280)
        return {"kind": kind, "scene": rng.choice(["spheres", "mixed", "heightfield"]), "tris": _log(rng, 20000, 300000),
                "w": w, "h": int(w * 0.5625) + rng.randint(0, 5), "bvh": 2}
    if kind == "trace":
        return {"kind": kind, "tris": _log(rng, 16384, 131072), "n": _log(rng, 10000, 1200000)}
    if kind == "bake":
        ow = 2 ** rng.randint(5, 9)
        return {"kind": kind, "ow": ow, "oh": max(16, ow // rng.choice([1, 2, 4])), "samples": rng.randint(16, 128),
                "sw": _log(rng, 256, 2048), "sh": _log(rng, 128, 1024), "ch": rng.choice([3, 4])}
    if kind == "command":
        ow = 2 ** rng.randint(5, 8)
        sw = _log(rng, 256, 1024)
        return {"kind": kind, "ow": ow, "oh": ow // 2, "samples": rng.randint(16, 128), "sw": sw, "sh": sw // 2 + 1}
    w = _log(rng, 320, 3840)
    h = int(w * 0.5625) + rng.randint(0, 7)
    return {"kind": "film", "w": w, "h": h, "ch": rng.choice([3, 4]), "dw": max(64, int(w * rng.uniform(0.2, 1.0))),
            "dh": max(64, int(h * rng.uniform(0.2, 1.0)))}


# ---------------------------------------------------------------- scenes


def _scene(name, tris, w, h, seed):
    if name == "spheres":  # spheres of 1024 triangles on the ground
        return scenes.spheres_scene(w, h, n_spheres=max(1, tris // 1024), seed=seed)
    if name == "mixed":
        return scenes.mixed_scene(tris, w, h, seed=seed)
    if name == "heightfield":
        return scenes.heightfield_scene(n=max(8, int(round(math.sqrt(tris / 2.0)))), width=w, height=h, env_w=1024,
                                        env_h=512, seed=seed)
    # 10 meshes, 1000 instances
    return scenes.instanced_scene(n_meshes=10, n_instances=1000, tris_per_mesh=max(64, tris // 1000), width=w, height=h,
                                  seed=seed, env_w=1024, env_h=512)


def _pinned(scene):
    """The scene with its arrays in pinned host memory, as a program that uploads often keeps them."""
    def pin(a):
        return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()

    out = dict(scene)
    out["meshes"] = [{k: pin(v) for k, v in m.items()} for m in scene["meshes"]]
    out["textures"] = [dict(t, pixels=pin(t["pixels"])) for t in scene["textures"]]
    return out


def _ready(scene, bvh=2):
    ctx = native.Context(0)
    ctx.upload(scene)
    ctx.build(width=bvh)
    return ctx


def _job_list(case, seed):
    """The frames of a batch: square films between a third of `side` and `side`, samples and depths
    up to the case's (the case's own; the seed picks the scenes' contents and the samplers)."""
    rng = np.random.default_rng([case["jobs"], case["tris"], case["side"], case["spp"], case["depth"]])
    jobs = []
    for j in range(case["jobs"]):
        side = int(round(math.exp(rng.uniform(math.log(case["side"] / 3.0), math.log(case["side"])))))
        tris = int(rng.integers(case["tris"] // 4, case["tris"] + 1))
        spp = max(1, case["spp"] // int(rng.choice([1, 2, 4])))
        depth = max(2, case["depth"] // int(rng.choice([1, 2, 4])))
        jobs.append((side, tris, spp, depth, seed * 1000 + j))
    return jobs


def _film(w, h):
    return torch.empty((h, w, 4), dtype=torch.float32, device="cuda")


# ---------------------------------------------------------------- prepare / run


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "frame":
        scene = _scene(case["scene"], case["tris"], case["w"], case["h"], seed)
        s["ctx"] = _ready(scene, case["bvh"])
        s["frame"] = native.make_frame(scene, case["w"], case["h"], case["spp"], case["depth"], seed=seed,
                                       rr_start=case["rr"])
        s["film"] = _film(case["w"], case["h"])
    elif kind in ("batch", "pipeline"):
        jobs = _job_list(case, seed)
        made = [_scene("mixed", t, side, side, q) for side, t, _, _, q in jobs]
        s["frames"] = [native.make_frame(sc, side, side, spp, depth, seed=q)
                       for sc, (side, _, spp, depth, q) in zip(made, jobs)]
        if kind == "batch":
            s["ctxs"] = [_ready(sc) for sc in made]
            s["films"] = [_film(j[0], j[0]) for j in jobs]
        else:
            s["ctxs"] = [native.Context(0) for _ in jobs]
            s["scenes"] = [native.prepare_scene(_pinned(sc)) for sc in made]
            s["films"] = [torch.empty((j[0], j[0], 4), dtype=torch.float32).pin_memory().numpy() for j in jobs]
    elif kind == "adjoint":
        scene = _scene("spheres", case["tris"], case["w"], case["h"], seed)
        s["ctx"] = _ready(scene)
        s["frame"] = native.make_frame(scene, case["w"], case["h"], case["spp"], case["depth"], seed=seed)
        s["film"] = _film(case["w"], case["h"])
        n, m = s["ctx"].info()["triangles"], len(scene["materials"])
        s["albedo"] = torch.rand((n, 3), generator=gen, device="cuda") * 0.6 + 0.2
        s["rough"] = torch.rand((m,), generator=gen, device="cuda") * 0.7 + 0.2
        s["target"] = torch.rand((case["h"], case["w"], 4), generator=gen, device="cuda")
    elif kind == "edit":
        scene = _scene(case["scene"], case["tris"], case["w"], case["h"], seed)
        s["ctx"] = native.Context(0)
        s["scene"] = native.prepare_scene(_pinned(scene))
        s["bvh"] = case["bvh"]
        s["frame"] = native.make_frame(scene, case["w"], case["h"], 1, 1, seed=seed)
        s["depth"], s["normal"] = _film(case["w"], case["h"]), _film(case["w"], case["h"])
    elif kind == "trace":
        s["ctx"] = _ready(_scene("spheres", case["tris"], 256, 256, seed))
        s["o"], s["d"] = _rays(case, gen)
        n = case["n"]
        s["prim"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["t"], s["u"], s["v"] = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(3))
    elif kind == "bake":
        s["ctx"] = native.Context(0)
        s["src"] = _environment(case, case["ch"], gen)
        s["out"] = torch.zeros((case["oh"], case["ow"], case["ch"]), dtype=torch.float32, device="cuda")
        s["case"] = case
    elif kind == "command":
        s["ctx"] = native.Context(0)
        s["dir"] = _Folder()
        s["in"], s["out"] = os.path.join(s["dir"].path, "env"), os.path.join(s["dir"].path, "irradiance")
        s["ctx"].hdr_write(s["in"], case["sw"], case["sh"], 4, pixels_host=_environment(case, 4, gen).cpu().numpy())
        s["case"] = case
    else:
        s["ctx"] = native.Context(0)
        shape = (case["h"], case["w"], case["ch"])
        s["partial"] = torch.randn(shape, generator=gen, device="cuda").exp_()
        s["accum"] = torch.randn(shape, generator=gen, device="cuda").exp_() * 7.0
        s["mean"], s["display"] = torch.empty(shape, device="cuda"), torch.empty(shape, device="cuda")
        # the snapshot writes three channels of each pixel: the rest is the program's own
        s["snap"] = torch.zeros((case["dh"], case["dw"], case["ch"]), device="cuda")
        s["case"] = case
    torch.cuda.synchronize()
    return s


class _Folder:
    """A temporary folder that goes with the state."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="nova_cases_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


def _rays(case, gen):
    """Incoherent rays: origins in the box above the ground, directions uniform on the sphere."""
    n = case["n"]
    o = torch.rand((n, 3), generator=gen, device="cuda") * torch.tensor([20.0, 4.0, 20.0], device="cuda") + torch.tensor(
        [-10.0, 0.05, -10.0], device="cuda")
    d = torch.randn((n, 3), generator=gen, device="cuda")
    return o.contiguous(), (d / d.norm(dim=1, keepdim=True)).contiguous()


def _environment(case, ch, gen):
    """A smooth sky with a bright log-normal texture, as a captured environment has."""
    h, w = case["sh"], case["sw"]
    e = torch.randn((h, w, ch), generator=gen, device="cuda").mul_(0.5).exp_()
    y = torch.linspace(0.0, 1.0, h, device="cuda").view(h, 1, 1)
    return (e * (0.2 + 2.0 * (1.0 - y))).contiguous()


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["ctx"].render(s["frame"], film_device_ptr=s["film"].data_ptr())
        return s["film"]
    if kind == "batch":
        native.render_batch(s["ctxs"], s["frames"], films_device=[f.data_ptr() for f in s["films"]])
        return s["films"]
    if kind == "pipeline":
        native.upload_build_render_batch(s["ctxs"], s["scenes"], s["frames"], films_host=s["films"])
        return s["films"]
    if kind == "adjoint":
        ctx = s["ctx"]
        g_alb, g_rough = torch.zeros_like(s["albedo"]), torch.zeros_like(s["rough"])
        ctx.set_diff_params(s["albedo"].data_ptr(), s["rough"].data_ptr())
        ctx.render(s["frame"], film_device_ptr=s["film"].data_ptr())
        d_image = (s["film"] - s["target"]) * (2.0 / s["film"].numel())
        torch.cuda.current_stream().synchronize()  # the library works on its own stream
        ctx.backward(s["frame"], d_image.data_ptr(), g_alb.data_ptr(), g_rough.data_ptr(), reuse_primal=True)
        ctx.set_diff_params(None, None)
        return {"film": s["film"], "albedo": g_alb, "roughness": g_rough}
    if kind == "edit":
        ctx = s["ctx"]
        ctx.upload(s["scene"])
        ctx.build(width=s["bvh"])
        ctx.render_aov(s["frame"], native.AOV_DEPTH, 0.1, 1000.0, film_device_ptr=s["depth"].data_ptr())
        ctx.render_aov(s["frame"], native.AOV_NORMAL, film_device_ptr=s["normal"].data_ptr())
        return {"depth": s["depth"], "normal": s["normal"]}
    if kind == "trace":
        s["ctx"].trace(s["o"].data_ptr(), s["d"].data_ptr(), s["t"].numel(), s["prim"].data_ptr(), s["t"].data_ptr(),
                       s["u"].data_ptr(), s["v"].data_ptr())
        return {"prim": s["prim"], "t": s["t"], "u": s["u"], "v": s["v"]}
    if kind == "bake":
        c = s["case"]
        s["ctx"].bake_irradiance(s["src"].data_ptr(), c["sw"], c["sh"], c["ch"], c["ow"], c["oh"], c["samples"],
                                 s["out"].data_ptr())
        return s["out"]
    if kind == "command":
        c = s["case"]
        s["ctx"].bake_texture("irradiance", c["ow"], c["oh"], c["samples"], s["in"] + ".hdr", s["out"], gpu_kernel=True)
        # the file's bytes; its length depends on the run-length packing, so zeros follow up to the most
        data = np.fromfile(s["out"] + ".hdr", np.uint8)
        whole = np.zeros(128 + c["oh"] * 4 * (c["ow"] + c["ow"] // 64 + 9), np.uint8)
        whole[:data.size] = data
        return whole
    c, ctx = s["case"], s["ctx"]
    n = c["w"] * c["h"] * c["ch"]
    ctx.film_accumulate(s["partial"].data_ptr(), s["accum"].data_ptr(), s["mean"].data_ptr(), n, 7)
    ctx.display_blend(s["partial"].data_ptr(), s["accum"].data_ptr(), s["display"].data_ptr(), n, 7)
    ctx.snapshot(s["mean"].data_ptr(), c["w"], c["h"], c["ch"], s["snap"].data_ptr(), c["dw"], c["dh"])
    return {"accum": s["accum"], "mean": s["mean"], "display": s["display"], "snapshot": s["snap"]}


# ---------------------------------------------------------------- work


def _scene_bytes(tris):
    """One triangle's indices and its share of the vertices (64 B records, about one vertex for two
    triangles), and its share of the tree."""
    return 12.0 * tris + 32.0 * tris + 64.0 * tris


def _path_flops(paths, tris, depth):
    """A path of about min(depth + 1, 2.5) segments; per segment one descent of a binary tree (two
    boxes of 12 operations a level), one triangle test (about 45) and one scattering event (about 300)."""
    return paths * min(depth + 1, 2.5) * (24.0 * math.log2(max(tris, 2)) + 45.0 + 300.0)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        px = case["w"] * case["h"]
        unique = case["tris"] // 100 if case["scene"] == "instanced" else case["tris"]
        return {"bytes": _scene_bytes(unique) + 16.0 * px, "flops": _path_flops(px * case["spp"], case["tris"], case["depth"])}
    if kind in ("batch", "pipeline"):
        # the mean film of a batch has about 0.4 side^2 pixels; samples and depth about 0.6 of the most
        px, tris = 0.4 * case["side"] ** 2 * case["jobs"], 0.6 * case["tris"]
        by = _scene_bytes(tris) * case["jobs"] + 16.0 * px
        if kind == "pipeline":
            by += 68.0 * tris * case["jobs"]  # the scene's arrays over the bus
        return {"bytes": by, "flops": _path_flops(px * 0.6 * case["spp"], tris, 0.6 * case["depth"])}
    if kind == "adjoint":
        px = case["w"] * case["h"]
        # film and image gradient; parameters read, gradients written; forward and replay
        return {"bytes": _scene_bytes(case["tris"]) + 32.0 * px + 24.0 * case["tris"],
                "flops": 2.0 * _path_flops(px * case["spp"], case["tris"], case["depth"])}
    if kind == "edit":
        px = case["w"] * case["h"]
        return {"bytes": 2.0 * _scene_bytes(case["tris"]) + 32.0 * px,
                "flops": 2.0 * px * (24.0 * math.log2(case["tris"]) + 45.0) + case["tris"] * 50.0 * math.log2(case["tris"])}
    if kind == "trace":
        return {"bytes": _scene_bytes(case["tris"]) + 40.0 * case["n"],
                "flops": case["n"] * (24.0 * math.log2(case["tris"]) + 45.0)}
    if kind in ("bake", "command"):
        src, out = case["sw"] * case["sh"], case["ow"] * case["oh"]
        return {"bytes": (16.0 + (4.0 if kind == "command" else 0.0)) * (src + out),
                "flops": out * case["samples"] * 120.0}
    n, m = case["w"] * case["h"] * case["ch"], case["dw"] * case["dh"] * 3
    # partial and sum read, sum and mean written; partial and sum read, display written; snapshot
    return {"bytes": 4.0 * (4 * n + 3 * n + 2 * m), "flops": 7.0 * n}


# ---------------------------------------------------------------- 64-bit values


def _closest(scene, o, d):
    """Closest hit (t, u, v) of every ray on the scene's world-space triangles (identity instances), in
    64 bits: the Moller-Trumbore determinants as products of Pluecker-like rows; misses are 0, -1."""
    tri = []
    for m in scene["meshes"]:
        tri.append(np.asarray(m["vertices"]).reshape(-1, 3)[np.asarray(m["indices"]).reshape(-1, 3).astype(np.int64)])
    tri = torch.from_numpy(np.concatenate(tri)).cuda().double()
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    k0 = (v0 * nrm).sum(1)
    bu = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1).T.contiguous()
    bv = torch.cat([-e1, -torch.linalg.cross(v0, e1)], 1).T.contiguous()
    o, d = o.double(), d.double()
    ray = torch.cat([torch.linalg.cross(o, d), d], 1)
    n = o.shape[0]
    t, u, v = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3))
    hit = torch.zeros(n, dtype=torch.bool, device="cuda")
    step = max(1, int(5e8) // tri.shape[0])
    for b in range(0, n, step):
        e = min(n, b + step)
        inv = 1.0 / -(d[b:e] @ nrm.T)
        uu = (ray[b:e] @ bu) * inv
        vv = (ray[b:e] @ bv) * inv
        tt = (o[b:e] @ nrm.T - k0) * inv
        bad = (uu < 0) | (vv < 0) | (uu + vv > 1) | (tt < 1e-6) | ~torch.isfinite(tt)
        best, at = tt.masked_fill_(bad, math.inf).min(1)
        row = torch.arange(e - b, device="cuda")
        ok = torch.isfinite(best)
        hit[b:e] = ok
        zero = torch.zeros_like(best)
        t[b:e], u[b:e], v[b:e] = (torch.where(ok, x, zero) for x in (best, uu[row, at], vv[row, at]))
        del inv, uu, vv, tt, bad
    return hit, t, u, v


def _camera_rays(scene, w, h):
    """One unjittered camera ray per pixel, in 64 bits."""
    iP = torch.from_numpy(np.asarray(scene["inv_P"], np.float64).reshape(4, 4, order="F")).cuda()
    iV = torch.from_numpy(np.asarray(scene["inv_V"], np.float64).reshape(4, 4, order="F")).cuda()
    y, x = torch.meshgrid(torch.arange(h, device="cuda").double(), torch.arange(w, device="cuda").double(), indexing="ij")
    nx, ny = (2 * x - w) / w, (2 * y - h) / h
    one = torch.ones_like(nx)
    o = torch.stack([nx, ny, -one, one], -1).reshape(-1, 4) @ iP.T
    o = (o / o[:, 3:4])
    o[:, 3] = 1.0
    o = o @ iV.T
    d = torch.stack([nx, ny, -one, 0 * one], -1).reshape(-1, 4) @ iP.T
    d = torch.cat([d[:, :2], -torch.ones_like(d[:, 2:3]), torch.zeros_like(d[:, 3:4])], 1) @ iV.T
    d = d / d.norm(dim=1, keepdim=True)
    return o[:, :3].contiguous(), d[:, :3].contiguous()


def exact(case, seed):
    """Closest hits, depth images and film arithmetic in 64 bits.  A path's radiance has no such value:
    which lobe, texel and triangle it meets are discrete choices on the sampler's 32-bit hash, so
    another rounding is another path; an irradiance texel's hash seed is likewise the truncation of a
    32-bit approximation that lies on the boundary between two seeds."""
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if kind == "trace" and case["n"] * case["tris"] <= 1e11:
        scene = _scene("spheres", case["tris"], 256, 256, seed)
        _, t, u, v = _closest(scene, *_rays(case, gen))
        return {"prim": None, "t": t, "u": u, "v": v}
    if kind == "edit" and case["w"] * case["h"] * case["tris"] <= 1e11:
        scene = _scene(case["scene"], case["tris"], case["w"], case["h"], seed)
        hit, t, _, _ = _closest(scene, *_camera_rays(scene, case["w"], case["h"]))
        near, far = 0.1, 1000.0
        z = 1 - (t - near) / (far - near)
        z = (2 * near * far) / (far + near - z * (far - near)) * 2 - 1
        depth = torch.where(hit, z / far, torch.full_like(z, far))
        return {"depth": depth.view(case["h"], case["w"], 1).expand(-1, -1, 4).contiguous(), "normal": None}
    if kind == "film":
        shape = (case["h"], case["w"], case["ch"])
        partial = torch.randn(shape, generator=gen, device="cuda").exp_()
        accum = torch.randn(shape, generator=gen, device="cuda").exp_() * 7.0
        acc = accum.double() + partial.double()
        mean = acc / 8.0
        out = {"accum": acc, "mean": mean, "display": mean + 0.8 * (partial.double() - mean)}

        def pick(n, size):  # the texel a destination index reads: a 32-bit coordinate, truncated
            c = (np.arange(n, dtype=np.float64) / n).astype(np.float32) * np.float32(size)
            return torch.from_numpy(c.astype(np.int64)).cuda()

        snap = torch.zeros((case["dh"], case["dw"], case["ch"]), dtype=torch.float64, device="cuda")
        snap[..., :3] = mean[pick(case["dh"], case["h"])][:, pick(case["dw"], case["w"])][..., :3]
        out["snapshot"] = snap
        return out
    return None
