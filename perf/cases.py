"""Performance cases of the volumetric path tracer and its radiance cache.

Each case is one call (or the few calls of one frame) that a program of this framework makes:
plain launches of the tracer on a prepared scene, a radiance-cache frame, inference on a batch of
radiance queries, the training steps of one frame. `listed()` names them, `draw()` gives more of
the same ranges, `prepare()` makes what the program holds before the call, `run()` is the call,
`work()` what it cannot do without, `exact()` its values in 64 bits for the networks.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from rtc8_gb300 import nrc
from rtc8_gb300 import surfaces as surf
from rtc8_gb300._lib import check
from rtc8_gb300.configs import C1, C1_REFERENCE_MODE, C2, C5, C_ROOM, REFERENCE_RNG_SEED, VolumeSpec
from rtc8_gb300.convergence import NRC_SETTINGS
from rtc8_gb300.renderer import Renderer, device_view, setup_scene

ENCODINGS = {"reference": nrc.NRC_ENCODING_REFERENCE, "volume": nrc.NRC_ENCODING_VOLUME,
             "hashgrid": nrc.NRC_ENCODING_HASHGRID}


# ------------------------------------------------------------------------------ the cases
def plain(name, scene, width, height, spp, n, env, cell_log2):
    c = {"kind": "plain", "scene": scene, "width": width, "height": height, "spp": spp, "n": n, "env": env,
         "cell_log2": cell_log2}
    return dict(c, name=name) if name else c


def listed():
    return [
        # An interactive preview: one sample per pixel of the dense 64^3 cloud at 256^2, the
        # smallest launch a viewer issues while the camera moves.
        plain("preview_dense64_1spp", "dense", 256, 256, 1, 64, "constant", 3),
        # The dense configuration as it is rendered.
        plain("dense64_16spp", "dense", 256, 256, 16, 64, "constant", 3),
        # The benchmark's launch: sparse 512^3 cloud under the sky at 1024^2.
        plain("sparse512_16spp", "sparse", 1024, 1024, 16, 512, "sky", 5),
        # The largest scene: two unioned 1024^3 clouds at 2048^2, up to 1024 bounces.
        plain("stress1024_4spp", "union", 2048, 2048, 4, 1024, "sky", 6),
        # The reference's own path rules: per-pixel streams, one global majorant, no bounce cap.
        plain("reference_rules_8spp", "reference", 256, 256, 8, 64, "constant", 3),
        # Meshes around the cloud: the room (36 triangles) and the same with tessellated spheres,
        # which goes through the BVH.
        {"name": "room_4spp", "kind": "surface", "width": 512, "height": 512, "spp": 4, "n": 64, "segments": 0},
        {"name": "room_spheres_bvh_4spp", "kind": "surface", "width": 512, "height": 512, "spp": 4, "n": 64,
         "segments": 32},
        # A radiance-cache frame in the middle of a sequence: four training iterations and 128
        # samples per pixel, the whole pipeline.
        {"name": "cache_frame_256px", "kind": "frame", "width": 256, "height": 256, "spp": 128, "iterations": 4,
         "n": 64},
        # Inference on the queries of a 1024^2 render pass with the network of the reference's own
        # call (hash grid), and of a batched pass with the volume cache.
        {"name": "infer_hashgrid_1m", "kind": "infer", "encoding": "hashgrid", "records": 1 << 20},
        {"name": "infer_volume_4m", "kind": "infer", "encoding": "volume", "records": 1 << 22},
        # The four training steps of one training iteration (65,536 records), then the weights read
        # back as a program does that keeps or displays them.
        {"name": "train_hashgrid_64k", "kind": "train", "encoding": "hashgrid", "records": 65536},
        {"name": "train_volume_64k", "kind": "train", "encoding": "volume", "records": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "surface", "frame", "infer", "infer", "train"])
    if kind == "plain":
        scene = rng.choice(["dense", "dense", "sparse", "sparse", "reference"])
        if scene == "reference":
            width, height = _log(rng, 48, 320), _log(rng, 48, 320)
            spp, n = rng.randint(1, 8), _log(rng, 17, 160)
            return plain(None, scene, width, height, spp, n, rng.choice(["constant", "image"]), 3)
        width, height = _log(rng, 64, 1280), _log(rng, 64, 1280)
        n = _log(rng, 24, 160) if scene == "dense" else _log(rng, 96, 640)
        spp = max(1, min(_log(rng, 1, 32), 8_000_000 // (width * height)))
        cell = rng.randint(3, 4) if scene == "dense" else max(3, int(math.log2(n)) - 4 + rng.randint(0, 1))
        return plain(None, scene, width, height, spp, n, rng.choice(["constant", "sky", "image"]), cell)
    if kind == "surface":
        width, height = _log(rng, 64, 640), _log(rng, 64, 640)
        spp = max(1, min(rng.randint(1, 16), 1_000_000 // (width * height)))
        return {"kind": "surface", "width": width, "height": height, "spp": spp, "n": _log(rng, 24, 128),
                "segments": rng.choice([0, 0, 8, 16, 32, 64])}
    if kind == "frame":
        width, height = _log(rng, 96, 512), _log(rng, 96, 512)
        spp = max(1, min(_log(rng, 2, 128), 8_000_000 // (width * height)))
        return {"kind": "frame", "width": width, "height": height, "spp": spp, "iterations": rng.randint(1, 4),
                "n": _log(rng, 32, 128)}
    if kind == "infer":
        return {"kind": "infer", "encoding": rng.choice(list(ENCODINGS)), "records": _log(rng, 1000, 4_000_000)}
    return {"kind": "train", "encoding": rng.choice(list(ENCODINGS)), "records": 4 * _log(rng, 1000, 65536)}


# ------------------------------------------------------------------------------ scenes
def _config(case, seed):
    """The repository's configuration of the case's scene, with the case's sizes and the seed's
    cloud and random streams."""
    cloud = 1 + seed % 1_000_003
    kind = case["kind"]
    scene = case.get("scene", "dense")
    n = case["n"]
    if kind == "surface":
        base, vol = C_ROOM, VolumeSpec(n=n, seed=cloud, octaves=4, sigma_t_max=20.0)
    elif scene == "sparse":
        # Mean free paths in voxels as in the 512^3 configuration.
        octaves = max(4, min(6, int(math.log2(n)) - 3))
        base = C2
        vol = VolumeSpec(n=n, seed=cloud, octaves=octaves, threshold=0.55, sigma_t_max=200.0 * n / 512)
    elif scene == "union":
        base = C5
        vol = VolumeSpec(n=n, seed=cloud, octaves=6, threshold=0.78, sigma_t_max=400.0 * n / 1024,
                         union_seed=cloud + 1)
    elif scene == "reference":
        base, vol = C1_REFERENCE_MODE, VolumeSpec(n=n, seed=cloud, octaves=4, sigma_t_max=20.0)
    else:
        base, vol = C1, VolumeSpec(n=n, seed=cloud, octaves=4, sigma_t_max=20.0)
    cfg = base.replace(width=case["width"], height=case["height"], spp=case["spp"], volume=vol,
                       majorant_cell_log2=case.get("cell_log2", 3), rng_seed=REFERENCE_RNG_SEED + seed)
    env = case.get("env", "constant")
    if env == "sky":
        cfg = cfg.replace(sky=C2.sky, sun_elevation_deg=C2.sun_elevation_deg, env_constant=None)
    else:
        cfg = cfg.replace(sky=None, env_constant=0.5)
    return cfg


def _environment_image(seed):
    """A smooth HDR image with a bright lamp, as a light probe is."""
    rng = np.random.default_rng(seed)
    h, w = 200, 400
    y, x = np.mgrid[0:h, 0:w]
    img = np.zeros((h, w, 3), np.float32)
    for c in range(3):
        k = rng.uniform(1, 4, 2)
        img[..., c] = 0.4 + 0.3 * np.sin(2 * np.pi * x / w * round(k[0]) + c) * np.cos(np.pi * y / h * k[1])
    cy, cx = rng.integers(20, 90), rng.integers(20, w - 20)
    img[cy:cy + 6, cx:cx + 6] += 60.0
    return img


def _room(segments):
    """The room; with segments > 0 also two tessellated spheres (segments^2 triangles or so)."""
    sc = surf.room_scene()
    if segments:
        sc.add(surf.sphere(0.22, 5, segments, segments // 2), surf.translation(0.05, 0.05, 0.4))
        sc.add(surf.sphere(0.12, 4, segments, segments // 2), surf.translation(-0.35, 0.3, -0.2))
    return sc


def _scene_state(case, seed):
    cfg = _config(case, seed)
    r = Renderer(cfg.width, cfg.height)
    setup_scene(r, cfg)
    if case.get("env") == "image":
        r.set_environment_rgb(_environment_image(seed))
    if case["kind"] == "surface" and case["segments"]:
        r.set_surfaces(_room(case["segments"]))
    mean = ctypes.c_void_p()
    check(r.lib.vpt_get_accum_device_ptrs(r.ctx, None, ctypes.byref(mean)), "vpt_get_accum_device_ptrs")
    image = device_view(mean.value, (cfg.height, cfg.width, 3), "<f4")
    image.renderer = r  # the view is the renderer's memory: it keeps the renderer alive
    return {"kind": case["kind"], "renderer": r, "image": image, "spp": case["spp"]}


# ------------------------------------------------------------------------------ networks
def _queries(records, seed, encoding):
    """Radiance queries as the tracer writes them: a position in the world box, the polar angles of
    the normal and of the outgoing direction, roughness (the density in a medium), reflectances."""
    g = torch.Generator("cuda").manual_seed(seed)
    u = torch.rand((records, 14), generator=g, device="cuda")
    angles = torch.tensor([1, 1, 1, math.pi, 2 * math.pi, math.pi, 2 * math.pi] + [1] * 7, device="cuda")
    q = u * angles
    if encoding == "volume":  # a medium: normal = outgoing direction, diffuse = albedo, no specular
        q[:, 3:5] = q[:, 5:7]
        q[:, 8:11] = 0.99
        q[:, 11:14] = 0.0
    return q.contiguous()


def _targets(q):
    """A radiance field over the box with noise, non-negative as path estimates are."""
    p = q[:, :3]
    f = torch.stack([1.0 + torch.sin(5.0 * p[:, 0]) * torch.cos(3.0 * p[:, 1]), 0.6 + 0.4 * torch.sin(7.0 * p[:, 2]),
                     0.3 + p[:, 0] * p[:, 1]], 1)
    return (f * (0.5 + torch.roll(q[:, 7:8], 1, 0))).contiguous()


def _network(case, seed):
    """The cache of a program: the reference's settings for its encodings, the comparison's for the
    volume cache."""
    cfg = nrc.default_config(ENCODINGS[case["encoding"]])
    cfg.seed = 1 + seed % 1_000_003
    if case["encoding"] == "volume":
        cfg.learning_rate, cfg.ema_decay = NRC_SETTINGS["learning_rate"], NRC_SETTINGS["ema_decay"]
    cache = nrc.NeuralRadianceCache()
    cache.initialize(config=cfg)
    return cache


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("plain", "surface"):
        return _scene_state(case, seed)
    if kind == "frame":
        s = _scene_state(case, seed)
        r = s["renderer"]
        r.nrc_set_query_density(True)
        r.nrc_set_termination_factor(NRC_SETTINGS["termination"], NRC_SETTINGS["train_termination"])
        s["cache"] = _network({"encoding": "volume"}, seed)
        s["iterations"] = case["iterations"]
        # The sequence's first frame; the accumulation then starts anew.
        r.nrc_frame(s["cache"], NRC_SETTINGS["first_train_iterations"], case["spp"], True)
        r.reset_accumulation()
        return s
    cache = _network(case, seed)
    q = _queries(case["records"], seed, case["encoding"])
    s = {"kind": kind, "cache": cache, "queries": q, "records": case["records"]}
    if kind == "infer":
        if case["encoding"] == "hashgrid":  # table values of a trained cache's size
            p = cache.params()
            mlp = sum(a * b for a, b in zip(cache.layout()["in"], cache.layout()["out"]))
            p[mlp:] = np.random.default_rng(seed).standard_normal(p.size - mlp, dtype=np.float32) * np.float32(0.1)
            cache.set_params(p)
        s["out"] = torch.zeros((case["records"], 3), device="cuda")
    else:
        s["targets"] = _targets(q)
    return s


def run(state):
    kind = state["kind"]
    if kind in ("plain", "surface"):
        state["renderer"].launch_plain(state["spp"])
        return state["image"]
    if kind == "frame":
        state["renderer"].nrc_frame(state["cache"], state["iterations"], state["spp"], False)
        return state["image"]
    cache, q, n = state["cache"], state["queries"], state["records"]
    if kind == "infer":
        cache.infer(0, q, n, state["out"])
        return state["out"]
    step = n // 4
    for k in range(4):
        cache.train(0, q[k * step:], state["targets"][k * step:], step)
    return cache.params()


# ------------------------------------------------------------------------------ work and exact values
# Density lookups and path vertices per sample of the repository's configurations (its counters):
# what a sample's arithmetic follows from, about 40 operations a lookup and 200 a vertex.
PER_SAMPLE = {"dense": (4.2, 2.0), "sparse": (19.0, 2.4), "union": (9.8, 1.4), "reference": (10.1, 1.9),
              "surface": (18.0, 7.4)}


def _network_dims(encoding):
    return {"reference": (62, 2), "hashgrid": (58, 2), "volume": (138, 5)}[encoding]


def work(case):
    kind = case["kind"]
    if kind in ("plain", "surface", "frame"):
        pixels = case["width"] * case["height"]
        filled = {"dense": 1.0, "reference": 1.0, "sparse": 0.47, "union": 0.08}[case.get("scene", "dense")]
        texels = {"sky": 3200 * 1600, "image": 400 * 200}.get(case.get("env"), 64 * 32)
        lookups, vertices = PER_SAMPLE["surface" if kind == "surface" else case.get("scene", "dense")]
        samples = pixels * case["spp"]
        # Grid and environment read once; per pixel the random state, the sum in and out, the mean.
        w = {"bytes": 4.0 * filled * case["n"] ** 3 + 16.0 * texels + pixels * (8 + 48 + 12),
             "flops": samples * (40.0 * lookups + 200.0 * vertices)}
        if kind == "frame":
            t = work({"kind": "train", "encoding": "volume", "records": 65536})
            w = {k: w[k] + case["iterations"] * t[k] for k in w}
        return w
    inputs, hidden = _network_dims(case["encoding"])
    params = inputs * 64 + (hidden - 1) * 64 * 64 + 64 * 3
    grid = 0
    flops = 2.0 * params
    if case["encoding"] == "hashgrid":
        grid = 2 * sum(_grid_level(lv)[2] for lv in range(16))
        flops += 16 * 8 * 2 * 2
    n = case["records"]
    if kind == "infer":
        return {"bytes": n * (56.0 + 12.0) + 2.0 * (params + grid), "flops": n * flops}
    # Four steps: each reads its records and reads and writes weights, moments and average.
    return {"bytes": n * (56.0 + 12.0) + 4 * 32.0 * (params + grid), "flops": n * 3.0 * flops}


def _grid_level(lv):
    """(scale, resolution, entries, hashed) of a level of the reference's hash grid."""
    scale = 16.0 * 2.0 ** lv - 1.0
    res = math.ceil(scale) + 1
    entries = min((res ** 3 + 7) // 8 * 8, 1 << 15)
    return scale, res, entries, res ** 3 > entries


def _one_blob(x, bins):
    b = (torch.arange(bins, device=x.device, dtype=torch.float64) + 0.5) / bins
    return torch.exp(-0.5 * ((x[:, None] - b) * bins) ** 2)


def _encode(q, encoding, table):
    """The encoded inputs in 64 bits; `table` holds the hash grid's entries (pairs)."""
    p = q[:, :3]
    if encoding == "volume":
        a = math.pi * p[:, :, None] * 2.0 ** torch.arange(12, device=q.device, dtype=torch.float64)
        f = torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(len(q), 72)
        return torch.cat([f, _one_blob(q[:, 5] / math.pi, 32), _one_blob(q[:, 6] / (2 * math.pi), 32), q[:, 7:9]], 1)
    scales = (math.pi, 2 * math.pi, math.pi, 2 * math.pi, 1.0)
    rest = torch.cat([_one_blob(q[:, 3 + a] / s, 4) for a, s in enumerate(scales)] + [q[:, 8:14]], 1)
    if encoding == "reference":
        v = p[:, :, None] * 2.0 ** torch.arange(12, device=q.device, dtype=torch.float64)
        return torch.cat([(2.0 * (v - v.floor() - 0.5).abs()).reshape(len(q), 36), rest], 1)
    feats, off = [], 0
    for lv in range(16):
        scale, res, entries, hashed = _grid_level(lv)
        pos = scale * p.clamp(0, 1) + 0.5
        cell = pos.floor()
        frac, cell = pos - cell, cell.long()
        f = 0.0
        for c in range(8):
            bit = [(c >> d) & 1 for d in range(3)]
            x, y, z = (cell[:, d] + bit[d] for d in range(3))
            w = torch.ones_like(frac[:, 0])
            for d in range(3):
                w = w * (frac[:, d] if bit[d] else 1.0 - frac[:, d])
            if hashed:
                i = (x ^ ((y * 2654435761) & 0xFFFFFFFF) ^ ((z * 805459861) & 0xFFFFFFFF)) & (entries - 1)
            else:
                i = (x + (y + z * res) * res) % entries
            f = f + w[:, None] * table[off + i]
        feats.append(f)
        off += entries
    return torch.cat(feats + [rest], 1)


def _unpack(params, layout, encoding):
    """The weight matrices (real rows and columns) and the hash table, in 64 bits."""
    mats, at = [], 0
    inputs, _ = _network_dims(encoding)
    for j, (a, b) in enumerate(zip(layout["in"], layout["out"])):
        m = params[at:at + a * b].reshape(b, a)
        mats.append((at, a, b, m[:3 if j == layout["L"] - 1 else b, :inputs if j == 0 else a].clone()))
        at += a * b
    return mats, at, params[at:].reshape(-1, 2).clone()


def _forward(x, mats, exp):
    for m in mats[:-1]:
        x = torch.relu(x @ m.T)
    x = x @ mats[-1].T
    return torch.exp(x) if exp else x


def exact(case, seed):
    if case["kind"] not in ("infer", "train"):
        return None  # a path estimate: its values are those of its own random decisions
    enc = case["encoding"]
    s = prepare(case, seed)
    cfg, layout = s["cache"].config, s["cache"].layout()
    params = torch.from_numpy(s["cache"].params()).cuda().double()
    mats, nparams, table = _unpack(params, layout, enc)
    exp = cfg.output_activation == nrc.NRC_OUTPUT_EXP
    q = s["queries"]
    if case["kind"] == "infer":
        w = [m for _, _, _, m in mats]
        return torch.cat([_forward(_encode(c.double(), enc, table), w, exp) for c in q.split(1 << 17)])
    # Adam on the loss mean over records and channels of (y - t)^2 / (luminance(y)^2 + 0.01), the
    # denominator held constant.
    leaves = [m.requires_grad_() for _, _, _, m in mats] + ([table.requires_grad_()] if enc == "hashgrid" else [])
    first = [torch.zeros_like(v) for v in leaves]
    second = [torch.zeros_like(v) for v in leaves]
    step = case["records"] // 4
    for k in range(4):
        x, t = q[k * step:(k + 1) * step].double(), s["targets"][k * step:(k + 1) * step].double()
        y = _forward(_encode(x, enc, table), leaves[:len(mats)], exp)
        lum = (y.detach() * torch.tensor([0.2126, 0.7152, 0.0722], device="cuda", dtype=torch.float64)).sum(1)
        loss = ((y - t) ** 2 / (lum * lum + 0.01)[:, None]).mean()
        grads = torch.autograd.grad(loss, leaves)
        with torch.no_grad():
            for i, (v, g) in enumerate(zip(leaves, grads)):
                is_table = i >= len(mats)
                g = g if is_table else g + cfg.l2_reg * v
                on = g != 0 if is_table else torch.ones_like(g, dtype=torch.bool)
                m1 = cfg.beta1 * first[i] + (1 - cfg.beta1) * g
                m2 = cfg.beta2 * second[i] + (1 - cfg.beta2) * g * g
                first[i], second[i] = torch.where(on, m1, first[i]), torch.where(on, m2, second[i])
                d = first[i] / (1 - cfg.beta1 ** (k + 1)) / ((second[i] / (1 - cfg.beta2 ** (k + 1))).sqrt() + cfg.epsilon)
                v -= cfg.learning_rate * torch.where(on, d, torch.zeros_like(d))
    out = params.clone()
    for (at, a, b, _), m in zip(mats, leaves):
        out[at:at + a * b].view(b, a)[:m.shape[0], :m.shape[1]] = m.detach()
    if enc == "hashgrid":
        out[nparams:] = table.detach().reshape(-1)
    return out
