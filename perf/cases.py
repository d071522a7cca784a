"""The work a user of the framework has it do, as cases that can be timed.

listed() are the cases, draw() gives more of the same ranges; prepare() makes
what a user's program holds before a call (scenes on the device, ray sets,
images, networks), run() is one pass through the public entry points, work()
the bytes and operations a pass cannot do without, exact() the result in
64-bit arithmetic where there is one.

A path-traced image has no such value: each pixel is a sum over random paths
whose branches depend on the rounding of every step. Nearest hits, the
denoiser's image and its gradients have one.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vviewer_gb300 import Context, scenes
from vviewer_gb300.denoiser import Denoiser
from vviewer_gb300.renderer import RenderInfo

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # the viewer's preview while a scene is edited: a small image at few
        # samples, the buffers returned to the host; launches and latency count
        {"name": "render_preview", "kind": "render", "scene": "cornell", "freq": 0, "width": 256, "height": 256,
         "samples": 8, "depth": 8, "batch": 4, "option": "plain", "host": True},
        # the Cornell room at the size and sample count of the benchmark
        {"name": "render_cornell", "kind": "render", "scene": "cornell", "freq": 0, "width": 256, "height": 256,
         "samples": 64, "depth": 8, "batch": 4, "option": "plain", "host": True},
        # a final frame: participating medium, a million triangles, full HD
        # (fewer samples than a final frame's 256, the same kernels and pools)
        {"name": "render_medium", "kind": "render", "scene": "medium", "freq": 79, "width": 1920, "height": 1080,
         "samples": 32, "depth": 12, "batch": 4, "option": "plain", "host": False},
        # an open scene: hundreds of instances, many mesh lights, thin lens,
        # the sky importance sampled, at a size that no tile divides
        {"name": "render_sky", "kind": "render", "scene": "sky", "freq": 45, "width": 1919, "height": 1079,
         "samples": 16, "depth": 8, "batch": 4, "option": "env_is", "host": False},
        # the low-discrepancy sampler with the error-bar image, ragged size
        {"name": "render_pmj", "kind": "render", "scene": "random", "freq": 0, "width": 613, "height": 341,
         "samples": 18, "depth": 9, "batch": 3, "option": "pmj_m2", "host": True},
        # a render service: preview requests over several scenes, submitted
        # together, each waited for
        {"name": "jobs_mix", "kind": "jobs", "jobs": 12, "scenes": 3},
        # a scene handed over (acceleration structures built, uploaded) and
        # asked for the surfaces under a set of rays, as an editor does
        {"name": "upload_medium", "kind": "upload", "scene": "medium", "freq": 79, "rays": 4096},
        # visibility queries in bulk from a program on the host
        {"name": "rays_closest", "kind": "rays", "scene": "medium", "freq": 40, "rays": 1000003},
        # the denoiser on a preview
        {"name": "denoise_small", "kind": "denoise", "width": 256, "height": 256},
        # the denoiser on a 4K frame
        {"name": "denoise_4k", "kind": "denoise", "width": 3840, "height": 2160},
        # the denoiser's training: gradients of a batch of crops, and whole
        # optimiser steps at another batch shape
        {"name": "denoise_grads", "kind": "grads", "count": 8, "width": 256, "height": 256},
        {"name": "denoise_train", "kind": "train", "count": 3, "width": 336, "height": 208},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "jobs", "upload", "rays", "denoise", "denoise", "grads", "train"])
    if kind == "render":
        scene = rng.choice(["cornell", "medium", "sky", "random"])
        w, h = _log(rng, 64, 1920), _log(rng, 64, 1080)
        batch = rng.choice([1, 2, 3, 4, 8])
        most = max(1, min(64 // batch, 60_000_000 // (w * h * batch)))
        samples = batch * _log(rng, 1, most)
        option = rng.choice(["plain", "pmj_m2", "env_is"] if scene == "sky" else ["plain", "plain", "pmj_m2", "fp64"])
        freq = {"medium": _log(rng, 8, 79), "sky": _log(rng, 6, 45)}.get(scene, 0)
        return {"kind": kind, "scene": scene, "freq": freq, "width": w, "height": h, "samples": samples,
                "depth": rng.randint(3, 12), "batch": batch, "option": option, "host": rng.random() < 0.5}
    if kind == "jobs":
        return {"kind": kind, "jobs": rng.randint(2, 16), "scenes": rng.randint(1, 4)}
    if kind == "upload":
        return {"kind": kind, "scene": rng.choice(["medium", "random"]), "freq": _log(rng, 8, 79),
                "rays": _log(rng, 64, 16384)}
    if kind == "rays":
        return {"kind": kind, "scene": rng.choice(["medium", "random"]), "freq": _log(rng, 8, 60),
                "rays": _log(rng, 1000, 1000003)}
    if kind == "denoise":
        return {"kind": kind, "width": 16 * _log(rng, 4, 240), "height": 16 * _log(rng, 4, 135)}
    return {"kind": kind, "count": rng.randint(1, 8), "width": 16 * _log(rng, 4, 16), "height": 16 * _log(rng, 4, 16)}


# ---------------------------------------------------------------- inputs

_context = None


def context():
    """The program's one context, as long as it lives."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def _scene(case, seed):
    """(engine, render info) of a case's scene; the seed makes the scene."""
    w, h = case.get("width", 256), case.get("height", 256)
    kw = dict(seed=seed % 1000003 + 1, width=w, height=h, samples=case.get("samples", 4),
              depth=case.get("depth", 8), batch_size=case.get("batch", 4))
    if case["scene"] == "cornell":
        return scenes.cornell_box(**kw)
    if case["scene"] == "medium":
        return scenes.cornell_medium(freq=case["freq"], **kw)
    if case["scene"] == "sky":
        return scenes.instanced_sky_scene(freq=case["freq"], n_instances=256, sky_w=2048, sky_h=1024, **kw)
    engine = scenes.random_scene(kw["seed"], max_tris=200_000)
    return engine, RenderInfo(samples=kw["samples"], depth=kw["depth"], batch_size=kw["batch_size"], width=w,
                              height=h, write_files=False)


def _rays(n, seed):
    """Half of them a camera's rays into the room, half between random points
    of it, as visibility queries are: n x (origin, tmin, direction, tmax)."""
    g = np.random.default_rng(seed)
    o = g.uniform(0.02, 0.98, (n, 3))
    o[: n // 2] = (0.5, 0.5, 2.2)
    d = g.uniform(0.02, 0.98, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.empty((n, 8), dtype=np.float32)
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, 1e-3, d, 1e4
    return rays


def _images(case, seed):
    """Noisy radiance, albedo, normal and target images: smooth structure
    with heavy-tailed sampling noise on the radiance."""
    n, h, w = case.get("count", 1), case["height"], case["width"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def smooth(lo, hi):
        c = torch.rand((n, 4, max(2, h // 32), max(2, w // 32)), generator=g, device="cuda")
        c = torch.nn.functional.interpolate(c, size=(h, w), mode="bilinear", align_corners=True)
        return (lo + (hi - lo) * c).permute(0, 2, 3, 1).contiguous()

    target = smooth(0.0, 2.0)
    noise = torch.rand((n, h, w, 4), generator=g, device="cuda").clamp_(min=1e-6).log_().neg_()
    return (target * noise).contiguous(), smooth(0.0, 1.0), smooth(0.0, 1.0), target


# the network: (input channels, output channels) of its 3x3 convolutions
_CH = [32, 48, 64, 96, 128]


def _layers():
    out, prev = [], 16
    for c in _CH:
        out += [(prev, c), (c, c)]
        prev = c
    for k in (3, 2, 1, 0):
        out += [(_CH[k + 1] + _CH[k], _CH[k]), (_CH[k], _CH[k])]
    return out + [(_CH[0], 16)]


def _weights(seed):
    """He-initialised weights with small biases, as a trained network has."""
    g = np.random.default_rng(seed)
    parts, layers = [], _layers()
    for k, (cin, cout) in enumerate(layers):
        last = k == len(layers) - 1
        w = g.standard_normal((cout, 9 * cin)) * math.sqrt((0.3 if last else 2.0) / (9 * cin))
        b = g.standard_normal(cout) * 0.02
        if last:
            w[3:], b[3:] = 0.0, 0.0  # three radiance channels are used
        parts += [w.reshape(-1), b]
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    if kind == "render":
        engine, info = _scene(case, seed)
        flat = engine.scene.build()
        st = {"case": case, "gpu": ctx.upload(flat), "sd": engine.scene.scene_data(info.width, info.height),
              "info": info}
        if not case["host"]:
            names = ["radiance", "albedo", "normal"] + (["radiance_m2"] if case["option"] == "pmj_m2" else [])
            st["out"] = {k: torch.zeros((info.height, info.width, 4), device="cuda") for k in names}
        return st
    if kind == "jobs":
        g = np.random.default_rng(seed)
        pool = []
        for k in range(case["scenes"]):
            engine = scenes.random_scene(seed % 1000003 + 17 * k, max_tris=200_000)
            pool.append((engine, ctx.upload(engine.scene.build())))
        todo = []
        for k in range(case["jobs"]):
            engine, gpu = pool[int(g.integers(len(pool)))]
            w, h = scenes.SERVING_RESOLUTIONS[k % 2]
            spp = scenes.SERVING_SPPS[k // 2 % 3]
            todo.append((gpu, engine.scene.scene_data(w, h),
                         RenderInfo(samples=spp, depth=8, batch_size=4, width=w, height=h, write_files=False)))
        return {"case": case, "todo": todo}
    if kind in ("upload", "rays"):
        engine, _ = _scene(case, seed)
        st = {"case": case, "flat": engine.scene.build(), "rays": _rays(case["rays"], seed)}
        if kind == "rays":
            st["gpu"] = ctx.upload(st["flat"])
        return st
    images = _images(case, seed)
    dn = Denoiser(ctx, seed=1)
    dn.set_params(_weights(seed))
    if kind == "denoise":
        return {"case": case, "dn": dn, "images": [x[0].contiguous() for x in images[:3]],
                "out": torch.zeros((case["height"], case["width"], 4), device="cuda")}
    return {"case": case, "dn": dn, "images": images}


# ---------------------------------------------------------------- one pass


def _hits(h):
    return {"t": h["t"], "u": h["u"], "v": h["v"], "instance": h["instance"].view(np.int32),
            "primitive": h["primitive"].view(np.int32)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        option = case["option"]
        kw = dict(want_m2=option == "pmj_m2", env_is=option == "env_is",
                  sampler="pmj" if option == "pmj_m2" else "rtgems", reduce_fp64=option == "fp64")
        if case["host"]:
            r = state["gpu"].render(state["sd"], state["info"], **kw)
            out = {"radiance": r.radiance, "albedo": r.albedo, "normal": r.normal}
            return out | ({"m2": r.radiance_m2} if kw["want_m2"] else {})
        state["gpu"].render(state["sd"], state["info"], outputs={k: v.data_ptr() for k, v in state["out"].items()},
                            **kw)
        return state["out"]
    if kind == "jobs":
        jobs = [gpu.submit(sd, info) for gpu, sd, info in state["todo"]]
        out = []
        for j in jobs:
            r = j.result()
            out += [r.radiance, r.albedo, r.normal]
            j.release()
        return out
    if kind == "upload":
        gpu = context().upload(state["flat"])
        hits = gpu.trace_closest(state["rays"])
        gpu.release()
        return _hits(hits)
    if kind == "rays":
        return _hits(state["gpu"].trace_closest(state["rays"]))
    dn = state["dn"]
    if kind == "denoise":
        dn.apply(*state["images"], state["out"])
        return state["out"]
    if kind == "grads":
        loss, g = dn.gradients(*state["images"])
        return {"loss": loss, "grads": g}
    return {"loss": dn.train_step(*state["images"], lr=1e-3), "params": dn.params()}


# ---------------------------------------------------------------- what a pass cannot do without

# operations of one ray: about log2(triangles) boxes of 24, two triangles of
# 60; of one surface event with its light sample, about 400
_TRIANGLES = {"cornell": 36, "random": 60_000}


def _triangles(case):
    if case["scene"] == "medium":
        return 8 * 20 * case["freq"] ** 2
    if case["scene"] == "sky":
        return 8 * 20 * case["freq"] ** 2
    return _TRIANGLES[case["scene"]]


def _ray_flops(triangles):
    return 24.0 * math.log2(triangles + 2) + 120.0


def _network(pixels):
    """Multiply-adds of the network's convolutions over an image, times two,
    and its weights' bytes (float32)."""
    L, flops, level = _layers(), 0.0, [0, 0, 1, 1, 2, 2, 3, 3, 4, 4, 3, 3, 2, 2, 1, 1, 0, 0, 0]
    for (cin, cout), lv in zip(L, level):
        flops += 2.0 * 9 * cin * cout * pixels / 4 ** lv
    return flops, 4.0 * sum(9 * a * b + b for a, b in L)


def work(case):
    kind = case["kind"]
    if kind == "render":
        tris, pixels = _triangles(case), case["width"] * case["height"]
        paths = pixels * (case["samples"] // case["batch"]) * case["batch"]
        # an extension and a shadow ray per event, about three events a path
        images = 4 if case["option"] == "pmj_m2" else 3
        return {"bytes": 16.0 * images * pixels + 108.0 * tris,
                "flops": paths * 3.0 * (2 * _ray_flops(tris) + 400.0)}
    if kind == "jobs":
        paths = case["jobs"] * 163_840 * 18.7
        return {"bytes": 48.0 * 163_840 * case["jobs"] + case["scenes"] * 108.0 * 60_000,
                "flops": paths * 3.0 * (2 * _ray_flops(60_000) + 400.0)}
    if kind == "upload":
        tris = _triangles(case)
        # vertices and indices read, triangles and tree written; binning per level
        return {"bytes": tris * (46.0 + 12.0 + 48.0 + 32.0) + case["rays"] * 52.0,
                "flops": 30.0 * tris * math.log2(tris) + case["rays"] * _ray_flops(tris)}
    if kind == "rays":
        tris = _triangles(case)
        return {"bytes": case["rays"] * 52.0 + 48.0 * tris, "flops": case["rays"] * _ray_flops(tris)}
    pixels = case.get("count", 1) * case["width"] * case["height"]
    flops, weights = _network(pixels)
    if kind == "denoise":
        return {"bytes": 64.0 * pixels + weights, "flops": flops}
    # forward, input gradients, weight gradients; a training step also reads
    # and writes the parameters and the optimiser's two moments
    return {"bytes": 64.0 * pixels + 2 * weights + (6 * weights if kind == "train" else 0), "flops": 3 * flops}


# ---------------------------------------------------------------- 64 bits


def _nearest(flat, rays):
    """Distance of the nearest surface along each ray (tmax where there is
    none): every ray against every triangle, Moeller and Trumbore's test."""
    r = torch.from_numpy(rays).cuda().double()
    o, tmin, d, best = r[:, 0:3], r[:, 3:4], r[:, 4:7], r[:, 7].clone()
    for inst in flat.instances:
        if not inst.flags & 1:
            continue
        mesh = flat.meshes[inst.mesh_index]
        m = torch.tensor(list(inst.model), dtype=torch.float64, device="cuda").reshape(4, 4).T
        p = torch.from_numpy(np.ascontiguousarray(mesh.vertices["position"])).cuda().double()
        p = p @ m[:3, :3].T + m[:3, 3]
        tri = p[torch.from_numpy(mesh.indices.astype(np.int64)).cuda()]
        a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
        n = torch.linalg.cross(e1, e2)
        # with s = o - a and det = d.n: t = -s.n / det, u = (d x s).e2 / det,
        # v = -(d x s).e1 / det; every term a matrix product over rays and triangles
        od = torch.linalg.cross(d, o)
        a1, a2 = torch.linalg.cross(a, e1), torch.linalg.cross(a, e2)
        step = max(1, 48_000_000 // len(rays))
        for k in range(0, len(tri), step):
            s = slice(k, k + step)
            det = d @ n[s].T
            t = ((a[s] * n[s]).sum(1) - o @ n[s].T) / det
            u = (od @ e2[s].T - d @ a2[s].T) / det
            v = -(od @ e1[s].T - d @ a1[s].T) / det
            hit = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin)
            best = torch.minimum(best, torch.where(hit, t, math.inf).amin(1))
    return best


def _split(weights):
    out, at = [], 0
    for cin, cout in _layers():
        n = cout * 9 * cin
        out.append((weights[at:at + n].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2), weights[at + n:at + n + cout]))
        at += n + cout
    return out


def _forward(weights, radiance, albedo, normal):
    """The network's last layer, n x 16 x h x w."""
    F = torch.nn.functional
    P = _split(weights)

    def conv(k, x):
        y = F.conv2d(x, P[k][0], P[k][1], padding=1)
        return y if k == len(P) - 1 else F.relu(y)

    x = torch.cat([torch.log1p(radiance[..., :3].clamp(min=0)), albedo[..., :3], normal[..., :3]], -1)
    x = F.pad(x.permute(0, 3, 1, 2), (0, 0, 0, 0, 0, 7))
    e = []
    for lv in range(5):
        x = conv(2 * lv + 1, conv(2 * lv, F.avg_pool2d(x, 2) if lv else x))
        e.append(x)
    for k, lv in enumerate((3, 2, 1, 0)):
        x = torch.cat([F.interpolate(x, scale_factor=2, mode="nearest"), e[lv]], 1)
        x = conv(11 + 2 * k, conv(10 + 2 * k, x))
    return conv(18, x)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("upload", "rays"):
        if case["rays"] * _triangles(case) > 8e9:
            return None
        engine, _ = _scene(case, seed)
        t = _nearest(engine.scene.build(), _rays(case["rays"], seed))
        return {"t": t, "u": None, "v": None, "instance": None, "primitive": None}
    if kind not in ("denoise", "grads", "train"):
        return None
    if case.get("count", 1) * case["width"] * case["height"] > 2_500_000:
        return None
    radiance, albedo, normal, target = (x.double() for x in _images(case, seed))
    weights = torch.from_numpy(_weights(seed)).cuda().double().requires_grad_(kind != "denoise")
    y = _forward(weights, radiance, albedo, normal).permute(0, 2, 3, 1)[..., :3]
    if kind == "denoise":
        out = torch.ones((case["height"], case["width"], 4), dtype=torch.float64, device="cuda")
        out[..., :3] = torch.expm1(y[0].clamp(min=0))
        return out
    loss = (y - torch.log1p(target[..., :3].clamp(min=0))).abs().mean()
    loss.backward()
    g = weights.grad
    if kind == "grads":
        return {"loss": float(loss), "grads": g}
    # the optimiser's first step: moments start at zero, their bias corrected
    return {"loss": float(loss), "params": (weights - 1e-3 * g / (g.abs() + 1e-8)).detach()}
