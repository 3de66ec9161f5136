"""The work this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` says which public entry points a pass goes through:

  frame     Tracer.set_camera + Tracer.trace_device: one rendered frame of a scene that stays on the
            device (`cache` 0) or streams through the domain cache (`cache` = its share of the domains)
  views     Tracer.trace_views_device: several cameras, sizes and shaders in one batch
  scene     Tracer.set_scene + set_camera + trace_device: a new time step of a simulation (vertex
            normals, hierarchies, upload) and its first frame
  schedule  schedule_static: domain queues of the caller's own rays, without allocations
  score     mlp_forward: the domain proposal's scores for a batch of rays
  train     mlp_train: Adam steps of the domain proposal

Scenes are the wavelet isosurface grids of spray_gb300.scenes; a seed gives the camera orbit, the domain
albedos and (frame, views, scene) nothing else, so a mesh is generated once per shape.  Rays and training
pairs are drawn from the seed on the GPU.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import spray_gb300 as sg
from spray_gb300 import scenes

#: 22 domains per list and half the domains in the cache are the out-of-core workload's settings
_OOC_LIST = 22


def listed():
    return [
        # a thumbnail while a scene is set up: a dozen kernels per depth over a few thousand rays
        dict(name="thumbnail", kind="frame", shader="pt", light="point+diffuse", width=64, height=48, spp=2, bounces=3,
             area=2, rr=0, grid=2, mesh=24, materials=False, phases=False, cache=0.0, policy=0),
        # ambient occlusion of a 64-domain grid, eight bounded rays and a light ray per hit
        dict(name="ao_1024", kind="frame", shader="ao", light="point", width=1024, height=1024, spp=1, bounces=1,
             area=8, rr=0, grid=4, mesh=64, materials=False, phases=False, cache=0.0, policy=0),
        # the headline frame: path tracing, 16 samples, five bounces with Russian roulette
        dict(name="pt_1080p", kind="frame", shader="pt", light="quad", width=1920, height=1080, spp=16, bounces=5,
             area=1, rr=3, grid=4, mesh=64, materials=False, phases=False, cache=0.0, policy=0),
        # a ragged frame with mirrors, a specular lobe and two kinds of lights
        dict(name="pt_ragged", kind="frame", shader="pt", light="point+diffuse", width=853, height=477, spp=3, bounces=4,
             area=2, rr=0, grid=3, mesh=40, materials=True, phases=True, cache=0.0, policy=0),
        # an uneven batch of 24 views, half AO and half path tracing, 256 to 2048 pixels a side
        dict(name="views_24", kind="views", views=24, side=2048, spp=16, bounces=4, grid=4, mesh=64),
        # out of core in the reference's domain order (the default policy): bound by domain copies
        dict(name="ooc_reference", kind="frame", shader="pt", light="quad", width=1024, height=1024, spp=4, bounces=3,
             area=1, rr=0, grid=6, mesh=64, materials=False, phases=True, cache=0.5, policy=0),
        # out of core with batched passes
        dict(name="ooc_batched", kind="frame", shader="pt", light="quad", width=2048, height=2048, spp=8, bounces=4,
             area=1, rr=0, grid=6, mesh=96, materials=False, phases=True, cache=0.5, policy=2),
        # out of core with the trained proposal ordering the loads
        dict(name="ooc_learned", kind="frame", shader="pt", light="quad", width=1600, height=900, spp=4, bounces=4,
             area=1, rr=0, grid=6, mesh=64, materials=False, phases=True, cache=0.5, policy=3),
        # a simulation's next time step: 27 domains rebuilt and a first frame of them
        dict(name="scene_step", kind="scene", width=640, height=360, spp=1, bounces=2, grid=3, mesh=64),
        # a renderer without a device allocator queues its rays itself
        dict(name="queues", kind="schedule", rays=65521, grid=5),
        # proposal scores of a wavefront's rays
        dict(name="scores", kind="score", rays=1 << 20, grid=8),
        # a few optimiser steps of the proposal
        dict(name="train", kind="train", rays=262144, batch=65536, steps=8, grid=8),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["ooc"] * 2 + ["views", "scene", "schedule", "score", "train"])
    if kind in ("frame", "ooc"):
        ooc = kind == "ooc"
        shader = "pt" if ooc else rng.choice(["pt", "pt", "ao"])
        light = rng.choice(["point", "quad", "point+diffuse"])
        spp = _log(rng, 1, 16)
        side = _log(rng, 256 if ooc else 48, 1400 if ooc else 2048)
        # samples of a frame stay below the headline frame's
        side = min(side, int(math.sqrt((8 << 20 if ooc or shader == "ao" else 24 << 20) / spp)))
        return dict(kind="frame", shader=shader, light=light, width=side + rng.randrange(0, 33),
                    height=max(33, int(side * rng.uniform(0.5, 1.0))), spp=spp, bounces=1 if shader == "ao" else rng.randint(1, 5),
                    area=_log(rng, 1, 12) if shader == "ao" else rng.randint(1, 3), rr=rng.choice([0, 0, 2, 3]),
                    grid=rng.randint(4, 6) if ooc else rng.randint(1, 5), mesh=_log(rng, 24, 80),
                    materials=shader == "pt" and rng.random() < 0.3, phases=rng.random() < 0.5,
                    cache=rng.choice([0.25, 0.5, 0.75]) if ooc else 0.0, policy=rng.choice([0, 2, 2, 3, 4]) if ooc else 0)
    if kind == "views":
        return dict(kind="views", views=_log(rng, 2, 20), side=rng.choice([256, 512, 1024, 2048]), spp=rng.choice([1, 4, 16]),
                    bounces=rng.randint(1, 4), grid=rng.randint(2, 4), mesh=_log(rng, 24, 64))
    if kind == "scene":
        return dict(kind="scene", width=_log(rng, 64, 800), height=_log(rng, 64, 600), spp=rng.randint(1, 3),
                    bounces=rng.randint(1, 3), grid=rng.randint(1, 3), mesh=_log(rng, 16, 72))
    if kind == "schedule":
        return dict(kind="schedule", rays=_log(rng, 200, 65521), grid=rng.randint(1, 5))
    if kind == "score":
        return dict(kind="score", rays=_log(rng, 100, 1 << 20), grid=rng.randint(2, 8))
    batch = _log(rng, 500, 65536)
    return dict(kind="train", rays=batch * rng.randint(1, 4) + rng.randrange(0, 100), batch=batch, steps=rng.randint(1, 8),
                grid=rng.randint(2, 8))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _grid(grid, mesh, phases):
    """Meshes of a grid's domains in world space (they do not depend on the seed)."""
    return scenes.wavelet_grid(grid, mesh, colors="grey", light="point", phase_seed=2024 if phases else None)


def _scene(grid, mesh, phases, light, materials, seed):
    base = _grid(grid, mesh, phases)
    albedo = scenes.domain_albedo(len(base.domains), seed)
    kinds = np.random.default_rng(seed).integers(0, 4, len(base.domains)) if materials else np.zeros(len(base.domains), int)
    domains = []
    for d, a, k in zip(base.domains, albedo, kinds):
        colour = (int(a[0]) << 16) | (int(a[1]) << 8) | int(a[2])
        # a quarter of the domains are mirrors
        mirror = materials and k == 0
        domains.append(sg.Domain(d.vertices, d.faces, np.full(len(d.vertices), colour, np.uint32), d.bounds,
                                 1 if mirror else 0, (0.9, 0.9, 0.9) if mirror else (1, 1, 1)))
    return sg.Scene(domains, scenes.make_lights(light, *scenes.scene_box(base)))


def _frame_config(case, scene):
    ao = case["shader"] == "ao"
    cfg = dict(image_w=case["width"], image_h=case["height"], ao_mode=int(ao), ao_samples=case["area"],
               pixel_samples=case["spp"], bounces=case["bounces"], fov=60.0, rr_depth=case["rr"],
               schedule_policy=case["policy"])
    if ao:
        cfg.update(ao_max_distance=0.05 * scenes.scene_diagonal(scene), ao_light_shadow=1)
    if case["materials"]:
        cfg.update(ks=[0.2, 0.2, 0.2], shininess=8.0)
    if case["cache"]:
        cfg.update(cache_size=max(1, int(case["cache"] * len(scene.domains))), list_size=_OOC_LIST)
    if case["policy"] == 3:
        cfg.update(learn_frames=1, learn_samples=1 << 20)
    return cfg


def _prepare_frame(case, seed):
    scene = _scene(case["grid"], case["mesh"], case["phases"], case["light"], case["materials"], seed)
    tracer = sg.Tracer(_frame_config(case, scene))
    tracer.set_scene(scene)
    state = dict(tracer=tracer, camera=scenes.orbit_camera(scene, seed),
                 image=torch.zeros((case["height"], case["width"], 4), device="cuda"))
    if case["policy"] == 3:
        # the frame whose hits train the proposal
        tracer.set_camera(*scenes.orbit_camera(scene, seed, frame=1))
        tracer.trace_device(state["image"].data_ptr())
    return state


def _prepare_views(case, seed):
    scene = _scene(case["grid"], case["mesh"], False, "quad", False, seed)
    diag = scenes.scene_diagonal(scene)
    sides = [s for s in (256, 512, 1024, 2048) if s <= case["side"]]
    spps = [s for s in (1, 4, 16) if s <= case["spp"]]
    views = []
    for k in range(case["views"]):
        pos, look, up = scenes.orbit_camera(scene, seed, frame=k)
        side = sides[(k + k // 2) % len(sides)]  # every size under both shaders
        v = dict(position=pos, lookat=look, up=up, vfov=60.0, image_w=side, image_h=side,
                 pixel_samples=spps[k % len(spps)])
        if k % 2 == 0:
            v.update(ao_mode=1, ao_samples=8, bounces=1, ao_light_shadow=1, ao_max_distance=0.05 * diag, rr_depth=0)
        else:
            v.update(ao_mode=0, ao_samples=1, bounces=case["bounces"], rr_depth=3, ao_light_shadow=0, ao_max_distance=0.0)
        views.append(v)
    tracer = sg.Tracer(dict(image_w=256, image_h=256, ao_mode=0, ao_samples=1, pixel_samples=1, bounces=case["bounces"], fov=60.0))
    tracer.set_scene(scene)
    sizes = [v["image_w"] * v["image_h"] * 4 for v in views]
    return dict(tracer=tracer, views=views, sizes=sizes, image=torch.zeros(sum(sizes), device="cuda"))


def _prepare_scene(case, seed):
    scene = _scene(case["grid"], case["mesh"], False, "quad", False, seed)
    tracer = sg.Tracer(dict(image_w=case["width"], image_h=case["height"], ao_mode=0, ao_samples=1, pixel_samples=case["spp"],
                            bounces=case["bounces"], fov=60.0))
    return dict(tracer=tracer, scene=scene, camera=scenes.orbit_camera(scene, seed),
                image=torch.zeros((case["height"], case["width"], 4), device="cuda"))


def _boxes(grid):
    """Packed domain boxes of a grid over [-1, 1]^3, jittered inward: (grid^3, 6)."""
    rng = np.random.default_rng(grid)
    cell = 2.0 / grid
    ids = np.stack(np.meshgrid(*[np.arange(grid)] * 3, indexing="ij"), -1).reshape(-1, 3)
    lo = -1.0 + cell * ids
    lo_in, hi_in = rng.uniform(0.0, 0.1 * cell, (2, grid ** 3, 3))
    return np.concatenate([lo + lo_in, lo + cell - hi_in], 1).astype(np.float32)


def _rays(n, seed):
    """Half eye rays from an orbit position, half bounce rays from inside the grid."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((n, 6), generator=g, device="cuda")
    phi = 2.0 * math.pi * torch.rand((1,), generator=g, device="cuda")
    eye = torch.cat([4.0 * torch.sin(phi), 4.0 * torch.sin(phi * 0.0 + 0.5), 4.0 * torch.cos(phi)])
    inside = (torch.arange(n, device="cuda") >= n // 2)[:, None]
    org = torch.where(inside, 2.0 * u[:, :3] - 1.0, eye[None, :])
    target = 2.4 * u[:, 3:] - 1.2
    d = torch.where(inside, torch.randn((n, 3), generator=g, device="cuda"), target - org)
    return org.contiguous(), torch.nn.functional.normalize(d).contiguous()


def _samples(n, grid, seed):
    """Training pairs: rays, their first eight domains in entry order, the one that holds the hit."""
    boxes = torch.from_numpy(_boxes(grid)).cuda()
    org, d = _rays(n, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    near = torch.empty((n, 8), device="cuda")
    cand = torch.empty((n, 8), dtype=torch.int64, device="cuda")
    k = min(8, len(boxes))
    for i in range(0, n, 32768):  # slab tests of a block of rays with every box
        o, inv = org[i:i + 32768, None], 1.0 / d[i:i + 32768, None]
        a, b = (boxes[None, :, :3] - o) * inv, (boxes[None, :, 3:] - o) * inv
        t0, t1 = torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)
        t = torch.where((t0 <= t1) & (t1 > 1e-3), t0, torch.full_like(t0, math.inf))
        near[i:i + 32768, :k], cand[i:i + 32768, :k] = torch.topk(t, k, largest=False, sorted=True)
        near[i:i + 32768, k:], cand[i:i + 32768, k:] = math.inf, 0
    ncand = torch.isfinite(near).sum(1)
    cand = torch.where(torch.isfinite(near), cand, torch.zeros_like(cand))
    # the hit is in the nearest domain for about half of the rays; a tenth hits nothing
    r = torch.rand((n, 2), generator=g, device="cuda")
    label = torch.minimum((-torch.log2(r[:, 0].clamp_min(1e-6))).long(), ncand - 1)
    label = torch.where(r[:, 1] < 0.1, torch.full_like(label, -1), label)
    out = torch.zeros((n, 12), dtype=torch.int32, device="cuda")
    out[:, 0:3] = org.view(torch.int32)
    out[:, 3:6] = d.view(torch.int32)
    out[:, 6:10] = (cand[:, 0::2] | (cand[:, 1::2] << 16)).int()
    out[:, 10] = ncand.int()
    out[:, 11] = label.int()
    return out, boxes


_SHAPES = ((64, 64, 54, 64), (64, 64, 64, 64), (64, 64, 64, 64), (16, 64, 64, 8))  # rows, columns, inputs, outputs


def _params(seed):
    """He-uniform weights of the proposal's network, zero where the layout pads."""
    rng = np.random.default_rng(seed)
    parts = []
    for rows, cols, fan, outs in _SHAPES:
        w = np.zeros((rows, cols), np.float32)
        w[:outs, :fan] = rng.uniform(-1.0, 1.0, (outs, fan)) * math.sqrt(6.0 / fan)
        b = np.zeros(rows, np.float32)
        b[:outs] = rng.uniform(-0.05, 0.05, outs)
        parts += [w.reshape(-1), b]
    p = np.concatenate(parts)
    assert len(p) == sg.mlp_param_count()
    return torch.from_numpy(p).cuda()


_NORM = (0.0, 0.0, 0.0, 1.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        return dict(kind=kind, **_prepare_frame(case, seed))
    if kind == "views":
        return dict(kind=kind, **_prepare_views(case, seed))
    if kind == "scene":
        return dict(kind=kind, **_prepare_scene(case, seed))
    if kind == "schedule":
        org, d = _rays(case["rays"], seed)
        pad = lambda x: torch.cat([x, torch.zeros_like(x[:, :1])], 1).contiguous()
        capacity = min(1 << 20, 14 * case["rays"] + 64)
        return dict(kind=kind, boxes=torch.from_numpy(_boxes(case["grid"])).cuda(), org=pad(org), dir=pad(d), capacity=capacity,
                    entries=torch.zeros((capacity, 2), dtype=torch.int32, device="cuda"),
                    start=torch.zeros(case["grid"] ** 3 + 1, dtype=torch.int32, device="cuda"))
    samples, boxes = _samples(case["rays"], case["grid"], seed)
    state = dict(kind=kind, samples=samples, boxes=boxes, params=_params(seed), n=case["rays"])
    if kind == "score":
        state.update(logits=torch.zeros((case["rays"], 8), device="cuda"),
                     pred=torch.zeros(case["rays"], dtype=torch.int32, device="cuda"))
    else:
        state.update(m=torch.zeros_like(state["params"]), v=torch.zeros_like(state["params"]), done=0, batch=case["batch"],
                     steps=case["steps"], losses=torch.zeros(case["steps"], device="cuda"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "frame":
        state["tracer"].set_camera(*state["camera"])
        st = state["tracer"].trace_device(state["image"].data_ptr())
        return dict(image=state["image"], rays=[st["rays_primary"], st["rays_shadow"], st["rays_bounce"]])
    if kind == "views":
        st = state["tracer"].trace_views_device(state["views"], state["image"].data_ptr())
        return dict(images=list(torch.split(state["image"], state["sizes"])),
                    rays=[st["rays_primary"], st["rays_shadow"], st["rays_bounce"]])
    if kind == "scene":
        state["tracer"].set_scene(state["scene"])
        state["tracer"].set_camera(*state["camera"])
        st = state["tracer"].trace_device(state["image"].data_ptr())
        return dict(image=state["image"], rays=[st["rays_primary"], st["rays_shadow"], st["rays_bounce"]])
    if kind == "schedule":
        n = sg.schedule_static(state["boxes"].data_ptr(), len(state["boxes"]), state["org"].data_ptr(), state["dir"].data_ptr(),
                               len(state["org"]), 16, state["entries"].data_ptr(), state["capacity"], state["start"].data_ptr())
        return dict(entries=state["entries"], start=state["start"], count=n)
    if kind == "score":
        sg.mlp_forward(state["params"].data_ptr(), state["boxes"].data_ptr(), _NORM, state["samples"].data_ptr(), state["n"],
                       state["logits"].data_ptr(), state["pred"].data_ptr())
        return dict(logits=state["logits"], pred=state["pred"])
    sg.mlp_train(state["params"].data_ptr(), state["m"].data_ptr(), state["v"].data_ptr(), state["boxes"].data_ptr(), _NORM,
                 state["samples"].data_ptr(), state["n"], state["batch"], 1e-3, state["steps"], state["done"] + 1,
                 state["losses"].data_ptr())
    state["done"] += state["steps"]
    return dict(params=state["params"], m=state["m"], v=state["v"], losses=state["losses"])


# ------------------------------------------------------------------ bounds
def work(case):
    """Bytes: scene data or samples in, images, queues or scores out, once each.  Operations: every
    sample's camera ray and one box test, every score's and gradient's multiply-adds; the shadow and
    bounce rays and the walks depend on the scene and are left out."""
    kind = case["kind"]
    if kind in ("frame", "scene"):
        tris = case["grid"] ** 3 * 4.3 * case["mesh"] ** 2
        pixels = case["width"] * case["height"]
        # a triangle: 12 B of indices and half a vertex of 16 B
        return dict(bytes=20.0 * tris + 16.0 * pixels, flops=60.0 * pixels * case["spp"])
    if kind == "views":
        sides = [s for s in (256, 512, 1024, 2048) if s <= case["side"]]
        spps = [s for s in (1, 4, 16) if s <= case["spp"]]
        pixels = sum(sides[(k + k // 2) % len(sides)] ** 2 for k in range(case["views"]))
        tris = case["grid"] ** 3 * 4.3 * case["mesh"] ** 2
        return dict(bytes=20.0 * tris + 16.0 * pixels, flops=60.0 * pixels * sum(spps) / len(spps))
    if kind == "schedule":
        # 32 B per ray in; a line through a packed g^3 grid meets about 1.5 g domains, half of the rays start inside
        entries = case["rays"] * min(case["grid"] ** 3, 1.1 * case["grid"])
        return dict(bytes=32.0 * case["rays"] + 8.0 * entries + 24.0 * case["grid"] ** 3, flops=12.0 * entries)
    macs = 54 * 64 + 2 * 64 * 64 + 64 * 8
    if kind == "score":
        return dict(bytes=(48.0 + 32.0 + 4.0) * case["rays"], flops=2.0 * macs * case["rays"])
    rows = float(sum(min(case["batch"], case["rays"] - (k * case["batch"]) % case["rays"]) for k in range(case["steps"])))
    return dict(bytes=48.0 * rows + 3 * 2 * 54080.0 * case["steps"], flops=2.0 * rows * (3 * macs - 54 * 64))


# ------------------------------------------------------------------ values in 64 bits
def _features64(samples, boxes):
    f = samples.view(torch.float32)
    org, d = f[:, 0:3].double(), f[:, 3:6].double()
    cand = torch.stack([(samples[:, 6 + j // 2] >> (16 * (j % 2))) & 0xffff for j in range(8)], 1).long()
    ncand = samples[:, 10].long()
    present = torch.arange(8, device=samples.device)[None] < ncand[:, None]
    b = boxes.double()[cand]
    pc = 0.5 * (b[..., :3] + b[..., 3:]) - org[:, None]
    half = 0.5 * (b[..., 3:] - b[..., :3])
    along = (pc * d[:, None]).sum(-1)
    miss = ((pc * pc).sum(-1) - along * along).clamp_min(0).sqrt()
    r = (half * half).sum(-1).sqrt()
    per = torch.stack([along, miss, r, (miss / r).clamp_max(4), (along / r).clamp(-4, 4), torch.ones_like(r)], -1)
    return torch.cat([org, d, (per * present[..., None]).reshape(len(org), 48)], 1), present, samples[:, 11].long()


def _logits64(x, parts):
    for layer, (rows, cols, fan, outs) in enumerate(_SHAPES):
        w, b = parts[2 * layer].reshape(rows, cols)[:, :fan], parts[2 * layer + 1]
        x = x @ w.T + b
        x = x.clamp_min(0) if layer < 3 else x[:, :outs]
    return x


def _parts(p):
    return list(torch.split(p, [s for rows, cols, _, _ in _SHAPES for s in (rows * cols, rows)]))


def exact(case, seed):
    """Scores and training steps in 64 bits.  An image has no such value: which triangle a ray hits near
    an edge, and with it the rest of its path, is decided by the roundings of the 32-bit tests; queues
    are whole numbers and the bit patterns of entry distances."""
    if case["kind"] not in ("score", "train"):
        return None
    samples, boxes = _samples(case["rays"], case["grid"], seed)
    params = _params(seed).double()
    if case["kind"] == "score":
        out = []
        for i in range(0, case["rays"], 65536):
            x, present, _ = _features64(samples[i:i + 65536], boxes)
            out.append(torch.where(present, _logits64(x, _parts(params)), torch.full_like(x[:, :8], -math.inf)))
        return dict(logits=torch.cat(out), pred=None)
    n, batch = case["rays"], min(case["batch"], case["rays"])
    m, v, losses = torch.zeros_like(params), torch.zeros_like(params), []
    for k in range(case["steps"]):
        start = (k * batch) % n
        x, present, label = _features64(samples[start:start + batch], boxes)
        has = (label >= 0) & (label < present.sum(1))
        p = params.clone().requires_grad_(True)
        logits = torch.where(present, _logits64(x, _parts(p)), torch.full_like(x[:, :8], -math.inf))
        loss = torch.nn.functional.cross_entropy(logits[has], label[has])
        (g,) = torch.autograd.grad(loss, p)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        t = k + 1
        params = params - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
        losses.append(loss.detach())
    return dict(params=params, m=m, v=v, losses=torch.stack(losses))
