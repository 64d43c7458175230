"""The renders a user of this framework has it do, as timed cases over the public Python binding
(which is one ctypes call to each C entry point).

Each case names a way of using the library (`kind`) and the sizes of one call:

  tile      an interactive tile of one sample into host memory (the drop-in for rt_render_tile)
  frame     a film cleared, rendered to `spp` samples and read back into pinned memory
  viewport  the first image after the camera moved: one or a few samples and the 8-bit picture
  final     a studio still: samples with the guide passes taken on the way, denoised, 16-bit
  queue     camera x light-rig variants of one geometry through the batched queue
  adaptive  an adaptive render to a noise target, from the first round to convergence
  fit       one iteration of a fit: new parameters into the scene, then the adjoint
  denoise   the denoiser on host planes (the drop-in for rt_denoise_with)

Scenes are this package's own: `small` (5 k triangles), `studio` (HDRI, cut-outs, thin and clear
glass, coats, anisotropy), `lights` (every light kind), `knot` (a displaced torus knot of
2 seg_u seg_v triangles in 16 materials) and `instances` (10 k-triangle spheres placed 1000 times).
A seed gives the render seed, the camera's place and the lights' strength.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import repackshot_b200 as rtg
from repackshot_b200 import scenes

# ---- cases ------------------------------------------------------------------------------------------------


def listed():
    return [
        # One tile of an interactive refinement: the smallest call, where launches and allocations count.
        {"name": "tile_64", "kind": "tile", "scene": "small", "width": 256, "height": 256, "spp": 1, "depth": 8, "seg": 0, "tile": 64},
        # The small plain forward render: a thumbnail.
        {"name": "small_256_16spp", "kind": "frame", "scene": "small", "width": 256, "height": 256, "spp": 16, "depth": 8, "seg": 0},
        # A viewport after a camera move: a product at 720p, one sample, shown in 8 bits.
        {"name": "viewport_720p_1spp", "kind": "viewport", "scene": "knot", "width": 1280, "height": 720, "spp": 1, "depth": 12, "seg": 256},
        # The product still: the headline frame, the largest call.
        {"name": "frame_1080p_64spp", "kind": "frame", "scene": "knot", "width": 1920, "height": 1080, "spp": 64, "depth": 12, "seg": 512},
        # A cropped re-render at odd sizes with every light kind, a thin lens, the Blackman-Harris
        # filter and edge samples.
        {"name": "crop_617x351_7spp", "kind": "frame", "scene": "lights", "width": 617, "height": 351, "spp": 7, "depth": 10, "seg": 0},
        # A studio still with an HDRI and every kind of material, denoised for delivery.
        {"name": "studio_800x600_final", "kind": "final", "scene": "studio", "width": 800, "height": 600, "spp": 16, "depth": 12, "seg": 0},
        # 10 M instanced triangles (two levels), deep paths.
        {"name": "instances_1080p_4spp", "kind": "frame", "scene": "instances", "width": 1920, "height": 1080, "spp": 4, "depth": 16, "seg": 0},
        # A catalogue: 12 camera x light-rig variants of one product, uneven sizes and samples.
        {"name": "queue_12_jobs", "kind": "queue", "scene": "knot", "width": 1280, "height": 720, "spp": 16, "depth": 12, "seg": 256, "jobs": 12},
        # An adaptive render to a noise target: one full round, then ever fewer blocks.
        {"name": "adaptive_960x540", "kind": "adaptive", "scene": "knot", "width": 960, "height": 540, "spp": 64, "depth": 12, "seg": 256},
        # An iteration of the differentiable render at its own size, and of a coarse, odd-sized one.
        {"name": "fit_512_32spp", "kind": "fit", "scene": "fit", "width": 512, "height": 512, "spp": 32, "depth": 6, "seg": 0},
        {"name": "fit_203x97_5spp", "kind": "fit", "scene": "fit", "width": 203, "height": 97, "spp": 5, "depth": 6, "seg": 0},
        # The denoiser alone, on planes in host memory.
        {"name": "denoise_1280x720", "kind": "denoise", "scene": "planes", "width": 1280, "height": 720, "spp": 16, "depth": 0, "seg": 0, "preset": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tile", "frame", "frame", "frame", "viewport", "final", "queue", "adaptive", "fit", "denoise"])
    width = _log(rng, 64, 1920)
    height = max(48, min(1080, int(width * rng.uniform(0.5, 1.0))))
    c = {"kind": kind, "scene": "knot", "width": width, "height": height, "spp": 1, "depth": rng.randint(3, 16), "seg": rng.choice([16, 64, 256])}
    if kind == "tile":
        c["scene"] = rng.choice(["small", "studio", "lights"])
        c["tile"] = rng.randint(8, 48)
    elif kind == "frame":
        c["scene"] = rng.choice(["small", "studio", "lights", "knot", "instances"])
        c["spp"] = _log(rng, 1, max(2, min(128, 32_000_000 // (width * height))))
    elif kind == "viewport":
        c["scene"] = rng.choice(["small", "lights", "knot", "instances"])
        c["spp"] = rng.randint(1, 4)
    elif kind == "final":
        c["scene"] = rng.choice(["small", "studio", "lights"])
        c["spp"] = _log(rng, 4, max(5, min(64, 16_000_000 // (width * height))))
    elif kind == "queue":
        c["jobs"] = rng.randint(2, 12)
        c["spp"] = rng.choice([4, 16])
        c["width"], c["height"] = max(256, min(1280, width)), max(144, min(720, height))
    elif kind == "adaptive":
        c["width"], c["height"] = min(width, 960), min(height, 540)
        c["spp"] = rng.choice([24, 64])
    elif kind == "fit":
        c["scene"] = "fit"
        c["width"], c["height"] = min(width, 512), min(height, 512)
        c["spp"] = _log(rng, 2, 32)
        c["depth"] = rng.randint(3, 8)
    else:
        c.update(scene="planes", width=min(width, 1280), height=min(height, 720), spp=_log(rng, 1, 256), depth=0, preset=rng.randint(0, 1))
    if c["scene"] != "knot":
        c["seg"] = 0
    return c


# ---- scenes -------------------------------------------------------------------------------------------------


def _describe(case, seed, variant=0):
    """The case's scene: `variant` 0 is the one loaded, others are the queue's jobs over it."""
    g = random.Random(seed * 1009 + variant)
    w, h, spp, depth = case["width"], case["height"], case["spp"], case["depth"]
    kind = case["scene"]
    if kind == "knot":
        s = scenes.product_scene(width=w, height=h, spp=spp, depth=depth, seg_u=2 * case["seg"], seg_v=case["seg"],
                                 camera_angle_deg=g.uniform(-20.0, 20.0) + 45.0 * variant, focal_mm=50.0 if variant == 0 else g.uniform(35.0, 135.0),
                                 rig=scenes.light_rig(g.randint(0, 7)) if variant else None)
    elif kind == "instances":
        s = scenes.cfg4_scene(width=w, height=h, spp=spp, depth=depth)
    elif kind == "studio":
        s = scenes.e5_scene(sky=False)
        s.env_rotation = g.uniform(0.0, 60.0)
    elif kind == "lights":
        s = scenes.light_kinds_scene(w, h)
        s.fstop, s.pixel_filter, s.edge_supersample, s.clamp_indirect = 5.6, 3, 2, 20.0
    elif kind == "fit":
        s = scenes.adjoint_scene(w, h, spp, depth, perturb_seed=1 + seed % 1000)
    else:
        s = scenes.cfg0_scene()
    s.width, s.height, s.max_samples, s.max_depth = w, h, spp, depth
    s.seed = 1 + g.randrange(1 << 20)
    s.camera_position = tuple(c * g.uniform(0.98, 1.02) for c in s.camera_position)
    for light in s.lights:
        light.power *= g.uniform(0.9, 1.1)
    if case["kind"] == "adaptive":
        s.adaptive, s.noise_threshold = 1, 0.02
    return s


def _pinned(*shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _film_buffers(w, h):
    return (_pinned(3 * w * h), _pinned(w * h), _pinned(w * h), _pinned(w * h))


def _planes(case, seed):
    """Noisy sums of a scene of five balls before a wall over a floor, with their guide passes: the
    denoiser's 14 words a pixel (RGBA sums, squared luminance, albedo, normal, depth, part, material)."""
    w, h, n = case["width"], case["height"], case["spp"]
    g = torch.Generator().manual_seed(seed)
    y, x = torch.meshgrid(torch.arange(h, dtype=torch.float64) / h, torch.arange(w, dtype=torch.float64) / h, indexing="ij")
    part = torch.zeros(h, w, dtype=torch.int64)
    depth = torch.full((h, w), math.inf, dtype=torch.float64)
    normal = torch.zeros(h, w, 3, dtype=torch.float64)
    floor = y > 0.6
    part[floor] = 1
    depth[floor] = 1000.0 / (y[floor] - 0.4)
    normal[floor] = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64)
    for k in range(5):
        cx, cy, r = (torch.rand(3, generator=g, dtype=torch.float64) * torch.tensor([w / h, 0.8, 0.15]) + torch.tensor([0.0, 0.1, 0.08])).tolist()
        d2 = ((x - cx) ** 2 + (y - cy) ** 2) / (r * r)
        on = d2 < 1.0
        up = torch.sqrt((1.0 - d2).clamp(min=0.0))
        part[on] = k + 2
        depth[on] = (900.0 - 300.0 * r * up)[on]
        normal[on] = torch.stack([(x - cx) / r, -up, -(y - cy) / r], -1)[on]
    fg = part > 0
    colours = torch.rand(7, 3, generator=g, dtype=torch.float64) * 0.8 + 0.1
    albedo = colours[part] * fg[..., None]
    shade = 0.2 + 0.8 * (normal * torch.tensor([0.4, -0.5, 0.76], dtype=torch.float64)).sum(-1).clamp(min=0.0)
    mean = torch.where(fg[..., None], albedo * shade[..., None], torch.full((3,), 0.3, dtype=torch.float64))
    noise = 1.0 + 0.5 * torch.randn(h, w, generator=g, dtype=torch.float64).clamp(-1.9, 4.0) / math.sqrt(n)
    fire = torch.rand(h, w, generator=g) < 1.0e-4
    rgb = mean * torch.where(fire, 40.0, noise)[..., None] * n
    lum = (rgb * torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64)).sum(-1)
    lum2 = (lum * lum / n) * (1.0 + 0.25 * torch.rand(h, w, generator=g, dtype=torch.float64))
    sums = torch.cat([rgb, (fg * float(n))[..., None]], -1)
    f = lambda t: t.to(torch.float32).contiguous().numpy().reshape(-1).view(np.uint32)
    u = lambda t: t.to(torch.int32).contiguous().numpy().reshape(-1).view(np.uint32)
    return np.concatenate([f(sums), f(lum2), f(albedo), f(normal), f(depth), u(part), u(part)])


# ---- one case -------------------------------------------------------------------------------------------------


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, kind, w, h = case, case["kind"], case["width"], case["height"]
    if kind == "denoise":
        s.words = _planes(case, seed)
        return s
    desc = _describe(case, seed)
    s.scene = rtg.Scene(scenes.to_rsb(desc))
    if kind == "tile":
        g = random.Random(seed)
        t = case["tile"]
        s.rect = (g.randrange(max(1, w - t)), g.randrange(max(1, h - t)), t, t)
    elif kind == "queue":
        s.jobs = []
        for j in range(case["jobs"]):
            g = random.Random(31 + j)  # uneven sizes, the same for every seed
            c = dict(case, width=max(96, int(w * g.uniform(0.2, 1.0))), height=max(64, int(h * g.uniform(0.2, 1.0))), spp=max(1, case["spp"] >> g.randrange(3)))
            d = _describe(c, seed, 1 + j)
            s.jobs.append((scenes.to_rsb(d, meshes=False), c["spp"], c["width"], c["height"], _film_buffers(c["width"], c["height"])))
    elif kind == "fit":
        s.params = scenes.to_rsb(_describe(case, seed + 1), meshes=False)
        g = torch.Generator().manual_seed(seed)
        low = torch.rand(1, 3, 9, 9, generator=g) ** 2 * 1.5
        s.target = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear")[0].permute(1, 2, 0).contiguous().numpy()
        s.film = s.scene.film()
    else:
        s.film = s.scene.film()
        s.out = _film_buffers(w, h)
        if kind == "final":
            s.film.fuse_guides()
            s.clean = _pinned(h, w, 4)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "tile":
        return s.scene.render_tile(*s.rect, 0, rgba=True)
    if kind == "denoise":
        return rtg.denoise(s.words, s.case["width"], s.case["height"], s.case["spp"], preset=s.case["preset"])
    if kind == "queue":
        queue = rtg.Queue(s.scene)
        films = [queue.add(rsb, 0, spp, w, h) for rsb, spp, w, h, _ in s.jobs]
        queue.run()
        images = [film.read(job[4])[0] for film, job in zip(films, s.jobs)]
        for film in films:
            film.close()
        queue.close()
        return images
    if kind == "fit":
        s.scene.update(s.params)
        loss, grads, _ = s.scene.adjoint(s.film, s.target, 0, s.case["spp"])
        return {"loss": loss, "grads": grads}
    s.film.clear()
    if kind == "adaptive":
        render = rtg.Adaptive(s.scene, s.film, s.case["spp"])
        render.run()
        samples, _ = render.counts()
        render.close()
        return {"film": s.film.read(s.out), "samples": samples}
    if kind == "final":
        # the film's guide sums were cleared with it: the exact passes again, the albedo while rendering
        s.film.fuse_guides()
        s.film.render(0, s.case["spp"])
        s.film.denoise(s.case["spp"], out=s.clean)
        return {"film": s.film.read(s.out), "denoised": s.clean, "picture": s.film.srgb(bits=16)}
    s.film.render(0, s.case["spp"])
    if kind == "viewport":
        return {"film": s.film.read(s.out), "picture": s.film.srgb()}
    return s.film.read(s.out)


# ---- what a pass cannot do without --------------------------------------------------------------------------------

#: Triangles of the scenes whose count does not follow from the case, and mean rays a path (nearest
#: and any hit) of each scene at its usual depth, from the library's own ray counts.
TRIANGLES = {"small": 5122, "studio": 710, "lights": 710, "fit": 5122, "instances": 10002}
RAYS_PER_PATH = {"small": 3.3, "studio": 4.5, "lights": 3.5, "fit": 3.3, "instances": 4.5, "knot": 3.2}


def work(case):
    px, spp = case["width"] * case["height"], case["spp"]
    if case["kind"] == "denoise":
        # per pixel 56 bytes in, 16 out; 25 taps a level of about 60 operations, and as many again around them
        levels = 5 if case["preset"] == 0 else 3
        return {"bytes": px * 72.0, "flops": px * (levels * 25 * 60.0 + 300.0)}
    if case["kind"] == "tile":
        px = case["tile"] ** 2
    if case["kind"] == "queue":
        px, spp = case["jobs"] * px * 0.36, spp * 0.58
    if case["kind"] == "adaptive":
        spp *= 0.85
    tris = 4 * case["seg"] ** 2 if case["seg"] else TRIANGLES[case["scene"]]
    # a ray: the boxes of the nodes on its way down an eight-wide tree (8 boxes of 20 operations a
    # level, twice for the detours), three triangles of 50 operations; a vertex: about 600 operations
    ray = 2.0 * max(1.0, math.log(tris / 4.0, 8.0)) * 160.0 + 150.0
    rays = RAYS_PER_PATH[case["scene"]] * (2.0 if case["kind"] == "fit" else 1.0)
    # each triangle and vertex once, and the film out
    return {"bytes": tris * 48.0 + px * 24.0, "flops": px * spp * rays * (ray + 400.0)}


# ---- the denoiser in 64 bits ------------------------------------------------------------------------------------------


def exact(case, seed):
    """The denoised sums in 64 bits. The path tracer has no such value: a path in 64 bits takes other
    branches (lobes, roulette, which of two touching triangles) than one in 32, so its radiance is
    another sample and not this one's exact value; its films are compared bit for bit instead."""
    if case["kind"] != "denoise":
        return None
    w, h, n = case["width"], case["height"], case["spp"]
    words = _planes(case, seed)
    px = w * h
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    plane = lambda a, b: torch.from_numpy(words[a * px:b * px].view(np.float32).astype(np.float64)).to(dev).reshape(h, w, b - a)
    ids = lambda a: torch.from_numpy(words[a * px:(a + 1) * px].astype(np.int64)).to(dev).reshape(h, w)
    sums, lum2, albedo, normal, z = plane(0, 4), plane(4, 5)[..., 0], plane(5, 8), plane(8, 11), plane(11, 12)[..., 0]
    part, material = ids(12), ids(13)
    fg = part > 0
    y_lum = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=dev)
    lum = lambda c: (c * y_lum).sum(-1)

    def shifted(t, dx, dy, fill=0):
        out = torch.full_like(t, fill)
        x0, x1, y0, y1 = max(0, -dx), min(w, w - dx), max(0, -dy), min(h, h - dy)
        if x0 < x1 and y0 < y1:
            out[y0:y1, x0:x1] = t[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
        return out

    def same(dx, dy):
        return fg & (shifted(part, dx, dy, -1) == part) & (shifted(material, dx, dy, -1) == material)

    finite = torch.isfinite(z)

    def gradient(dx, dy):
        before, after = same(-dx, -dy) & shifted(finite, -dx, -dy, False), same(dx, dy) & shifted(finite, dx, dy, False)
        za, zb = shifted(z, -dx, -dy), shifted(z, dx, dy)
        zero = torch.zeros_like(z)
        return torch.where(finite & before & after, 0.5 * (zb - za), torch.where(finite & before, z - za, torch.where(finite & after, zb - z, zero)))

    gx, gy = gradient(1, 0), gradient(0, 1)
    divisor = torch.where(fg[..., None], albedo.clamp(min=0.01), torch.ones_like(albedo))
    mean = sums[..., :3] / n
    light = torch.where(fg[..., None], mean / divisor, torch.zeros_like(mean))
    var0 = torch.zeros_like(z)
    if n >= 4:
        l = lum(mean)
        var0 = torch.where(fg, (lum2 / n - l * l).clamp(min=0.0) / (n - 1) / lum(divisor) ** 2, var0)
    # fireflies: limited to four times their brightest neighbour; their variance is the largest about
    # them, an earlier firefly's as already replaced
    around = [(dx, dy) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if dx or dy]
    before = lum(light)
    brightest, count = torch.zeros_like(z), torch.zeros_like(part)
    for dx, dy in around:
        on = same(dx, dy)
        brightest = torch.where(on, torch.maximum(brightest, shifted(before, dx, dy)), brightest)
        count += on
    limit = 4.0 * brightest + 0.05
    fire = fg & (count >= 3) & (before > limit)
    light = torch.where(fire[..., None], light * (limit / before)[..., None], light)
    var = var0.clone()
    while True:
        swept = torch.zeros_like(z)
        for dx, dy in around:
            earlier = dy < 0 or (dy == 0 and dx < 0)
            v = shifted(torch.where(fire, var, var0) if earlier else var0, dx, dy)
            swept = torch.where(same(dx, dy), torch.maximum(swept, v), swept)
        swept = torch.where(fire, swept, var)
        if torch.equal(swept, var):
            break
        var = swept

    def depth_term(dx, dy):
        zq = shifted(z, dx, dy, math.inf)
        term = (z - zq).abs() / ((gx * dx + gy * dy).abs() + 1.0e-3 * z.abs() + 1.0e-6)
        flat = torch.where(z == zq, torch.zeros_like(z), torch.full_like(z, math.inf))
        return torch.where(finite & torch.isfinite(zq), term, flat)

    facing = lambda dx, dy: (normal * shifted(normal, dx, dy)).sum(-1).clamp(min=0.0) ** 128
    falloff = lambda e: (1.0 - e / 16.0).clamp(min=0.0) ** 16
    if n < 4:
        r = 3 if case["preset"] == 0 else 1
        sw, m1, m2 = torch.zeros_like(z), torch.zeros_like(z), torch.zeros_like(z)
        l = lum(light)
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                k = torch.where(same(dx, dy), facing(dx, dy) * falloff(depth_term(dx, dy)), torch.zeros_like(z))
                lq = shifted(l, dx, dy)
                sw, m1, m2 = sw + k, m1 + k * lq, m2 + k * lq * lq
        spread = (m2 / sw - (m1 / sw) ** 2).clamp(min=0.0)
        var = torch.where(fg & (sw > 0), spread, var)
    taps = (1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16)
    for level in range(5 if case["preset"] == 0 else 3):
        step = 1 << level
        l = lum(light)
        sw, sv = torch.zeros_like(z), torch.zeros_like(z)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = same(dx, dy) * ((2 - abs(dx)) * (2 - abs(dy)) / 16.0)
                sw, sv = sw + k, sv + k * shifted(var, dx, dy)
        blurred = torch.where(sw > 0, sv / sw, var)
        inv = 1.0 / (4.0 * torch.sqrt(blurred + 1.0e-10))
        sw, sv, sc = torch.zeros_like(z), torch.zeros_like(z), torch.zeros_like(light)
        for j in range(5):
            for i in range(5):
                dx, dy = (i - 2) * step, (j - 2) * step
                e = (l - shifted(l, dx, dy)).abs() * inv + depth_term(dx, dy) + (albedo - shifted(albedo, dx, dy)).abs().sum(-1) / 0.1
                wn = facing(dx, dy) if dx or dy else torch.ones_like(z)
                k = torch.where(same(dx, dy), taps[j] * taps[i] * wn * falloff(e), torch.zeros_like(z))
                sw, sv, sc = sw + k, sv + k * k * shifted(var, dx, dy), sc + k[..., None] * shifted(light, dx, dy)
        light = torch.where(fg[..., None], sc / sw[..., None], light)
        var = torch.where(fg, sv / (sw * sw), var)
    out = sums.clone()
    out[..., :3] = torch.where(fg[..., None], light * divisor * n, sums[..., :3])
    return out.reshape(-1).cpu().numpy()
