"""What the path tracer is measured on: whole calls of its public entry points
(render, batched render, scene creation, denoising, a denoiser training step,
tone mapping) on seeded synthetic scenes, with a context's default settings.

A case is a dict; "kind" says which entry point it stands for:

* box       the small Lambertian box (24 + 10 triangles): thumbnails and tests
* plugins   every material, light kind and texture slot in one small scene
* sky       three spheres under the analytic sun and sky
* mixed     N displaced icospheres of mixed materials under an environment map,
            thin lens: from an interactive frame to the 21M-triangle benchmark
* batch     several shots of one such scene in one render_batch call
* load      create_scene on host arrays, then the first preview frame
* denoise   a rendered film through the denoiser
* train     one training step (loss, gradients, Adam) on a batch of crops
* tonemap   a film's radiance through the post pass to a host image
"""
import functools
import math

import numpy as np
import torch

import asuna_gb300 as ag
from asuna_gb300 import _abi as A
from asuna_gb300 import denoise as dn
from asuna_gb300 import scenes

FILM_IMAGES = (0, 1, 2, 3, 8)  # radiance, albedo, normal, depth, filter-weight sum


def listed():
    return [
        # a thumbnail or a smoke test: a few thousand paths, launches and latency only
        {"name": "box_32x32x2", "kind": "box", "width": 32, "height": 32, "frames": 2, "depth": 8},
        # the default box render: a small scene at a moderate sample count
        {"name": "box_256x256x16", "kind": "box", "width": 256, "height": 256, "frames": 16, "depth": 8},
        # look development: every material, textured, with cut-out opacity
        {"name": "plugins_480x270x4", "kind": "plugins", "width": 480, "height": 270, "frames": 4, "depth": 8,
         "textured": True, "opacity": True},
        # an outdoor still at an odd size, procedural sky instead of a map
        {"name": "sky_641x427x8", "kind": "sky", "width": 641, "height": 427, "frames": 8, "depth": 6, "dusk": False},
        # one progressive frame of an interactive view, no Russian roulette
        {"name": "mixed_720p_1spp", "kind": "mixed", "width": 1280, "height": 720, "frames": 1, "depth": 8,
         "spheres": 16, "level": 6, "rr": 0},
        # the offline benchmark scene: 64 level-7 spheres, 1080p, depth 12, roulette after 3
        {"name": "mixed_1080p_8spp", "kind": "mixed", "width": 1920, "height": 1080, "frames": 8, "depth": 12,
         "spheres": 64, "level": 7, "rr": 3},
        # a turntable: 12 cameras around one scene, mixed sizes and sample counts, one call
        {"name": "batch_12_views", "kind": "batch", "shots": 12, "max_side": 512, "max_spp": 16, "depth": 12,
         "spheres": 8, "level": 7, "rr": 3},
        # opening a scene of 2M triangles: upload, acceleration structure, first preview
        {"name": "load_2M_preview", "kind": "load", "width": 320, "height": 180, "frames": 1, "depth": 8,
         "spheres": 24, "level": 6, "rr": 3},
        # the denoise pass of a finished 1080p still, default network
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080},
        # the denoise pass of a small preview at a size off the network's grid
        {"name": "denoise_251x187", "kind": "denoise", "width": 251, "height": 187},
        # one step of denoiser training, the training loop's default batch and crop
        {"name": "train_8x64", "kind": "train", "batch": 8, "crop": 64},
        # the 8-bit output path: post pass of a 1080p still, back on the host
        {"name": "tonemap_1080p", "kind": "tonemap", "width": 1920, "height": 1080, "operator": "filmic"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "plugins", "sky", "mixed", "mixed", "mixed", "batch", "load", "denoise", "train",
                       "tonemap"])
    c = {"kind": kind}
    if kind in ("box", "plugins", "sky", "mixed"):
        c["width"] = _log_int(rng, 24, 1920)
        c["height"] = max(16, int(c["width"] * rng.uniform(0.4, 1.0)))
        most = {"box": 1 << 21, "plugins": 1 << 20, "sky": 1 << 22, "mixed": 1 << 23}[kind]
        c["frames"] = _log_int(rng, 1, max(1, min(32, most // (c["width"] * c["height"]))))
        c["depth"] = rng.randint(3, 12)
    if kind == "plugins":
        c["textured"] = rng.random() < 0.5
        c["opacity"] = rng.random() < 0.5
    if kind == "sky":
        c["dusk"] = rng.random() < 0.5
    if kind == "load":
        c.update(width=_log_int(rng, 64, 640), height=_log_int(rng, 64, 360), frames=rng.randint(1, 2),
                 depth=rng.randint(3, 8))
    if kind in ("mixed", "load", "batch"):
        c["level"] = rng.randint(3, 7 if kind != "load" else 6)
        c["spheres"] = rng.randint(2, 24)
        c["rr"] = rng.choice([0, 3])
    if kind == "batch":
        c.update(shots=rng.randint(2, 12), max_side=_log_int(rng, 64, 512), max_spp=rng.choice([1, 4, 16]),
                 depth=rng.randint(3, 12))
    if kind in ("denoise", "tonemap"):
        c["width"] = _log_int(rng, 48, 1920)
        c["height"] = max(32, int(c["width"] * rng.uniform(0.4, 0.6)))
    if kind == "train":
        c.update(batch=rng.choice([4, 8, 16]), crop=rng.choice([32, 48, 64]))
    if kind == "tonemap":
        c["operator"] = rng.choice(["none", "gamma", "filmic", "aces", "pbrt"])
    return c


# ---- scenes -----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _icosphere(level):
    """Unit sphere: positions, faces, host indices, and each vertex's (at most
    six) faces, padded with the number of faces."""
    v, f = scenes.icosphere(level)
    faces = torch.from_numpy(f).cuda()
    flat = faces.reshape(-1)
    order = torch.argsort(flat, stable=True)
    count = torch.bincount(flat, minlength=len(v))
    slot = (torch.cumsum(count, 0) - count)[:, None] + torch.arange(6, device="cuda")
    around = torch.where(torch.arange(6, device="cuda") < count[:, None], order[slot.clamp_max(len(flat) - 1)] // 3,
                         len(f))
    return torch.from_numpy(v).cuda(), faces, f.astype(np.uint32).reshape(-1), around


def _displaced(level, seed):
    """A sphere mesh displaced by a seeded sum of plane waves, with
    area-weighted vertex normals (made on the GPU: there are many of them)."""
    base, faces, _, around = _icosphere(level)
    g = torch.Generator().manual_seed(seed)
    waves = (torch.randn(16, 3, generator=g, dtype=torch.float64) * 4.0).cuda()
    phase = (torch.rand(16, generator=g, dtype=torch.float64) * 6.2831853).cuda()
    pos = base * (1.0 + 0.0125 * torch.sin(base @ waves.T + phase).sum(1, keepdim=True))
    p = pos[faces]
    fn = torch.linalg.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    vn = torch.cat([fn, torch.zeros_like(fn[:1])])[around].sum(1)
    vn /= vn.norm(dim=1, keepdim=True).clamp_min(1e-30)
    v = np.zeros(len(base), A.VERTEX_DTYPE)
    v["pos"] = pos.float().cpu().numpy()
    v["normal"] = vn.float().cpu().numpy()
    return v


def _mixed_builder(spheres, level, seed):
    """The mixed-material recipe: 40% Lambertian, 40% rough plastic, 20%
    dielectric spheres in a 20^3 box over a ground quad, four triangle lights,
    a lognormal environment map with one bright spot."""
    rng = np.random.default_rng(seed)
    b = ag.SceneBuilder()
    for k in range(4):
        cx, cz = -6.0 + 4.0 * k, float(rng.uniform(-6, 6))
        b.add_triangle_light((cx - 1.2, 14.0, cz - 1.0), (cx, 14.0, cz + 1.4), (cx + 1.2, 14.0, cz - 1.0),
                             (40.0, 38.0, 34.0))
    b.set_envmap(scenes.lognormal_envmap(rng, 512, 256))
    ground = np.zeros(4, A.VERTEX_DTYPE)
    ground["pos"] = [(-40, -11, 40), (40, -11, 40), (40, -11, -40), (-40, -11, -40)]
    ground["normal"] = (0, 1, 0)
    b.add_mesh("ground", ground, np.array([0, 1, 2, 0, 2, 3], np.uint32))
    b.add_instance("ground", b.add_lambertian("ground", (0.5, 0.5, 0.5)))
    idx = _icosphere(level)[2]
    for k in range(spheres):
        u = rng.random()
        if u < 0.4:
            mat = b.add_lambertian(f"m{k}", rng.uniform(0.1, 0.9, 3))
        elif u < 0.8:
            a = float(rng.uniform(0.05, 0.8))
            mat = b.add_rough_plastic(f"m{k}", rng.uniform(0.1, 0.9, 3), (a, a), 1.5)
        else:
            mat = b.add_dielectric(f"m{k}", 1.5)
        b.add_mesh(f"sphere{k}", _displaced(level, seed + 31 * k), idx)
        # placed, turned about the vertical and, every third one, stretched
        t = scenes.rot_y(float(rng.uniform(0, 360)), rng.uniform(-10.0, 10.0, 3))
        if k % 3 == 0:
            t[:, 1] *= np.float32(rng.uniform(0.7, 1.4))
        elif k % 3 == 1:
            t[:, :3] = np.eye(3, dtype=np.float32)
        b.add_instance(f"sphere{k}", mat, t)
    return b


def _mixed_shot(b, case, width, height, frames, seed, eye=(0.0, 4.0, 30.0), at=(0.0, -2.0, 0.0)):
    return scenes.mixed_shot(b, width, height, frames, max_depth=case["depth"], rr_depth=case["rr"] or None, eye=eye,
                             at=at, seed=seed)


def _views(film, images=FILM_IMAGES):
    """The film's images as tensors; each keeps its film alive."""
    out = []
    for k in images:
        t = film.tensor(k)
        t.film = film
        out.append(t)
    return out


# ---- images of the denoiser and post cases ------------------------------------
def _images(seed, n, h, w):
    """Radiance with path-tracing noise (smooth shading times lognormal noise
    with a few fireflies), albedo and normal guides, filter-weight sums."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    y = torch.linspace(0, 1, h, device="cuda")[None, :, None, None]
    x = torch.linspace(0, 1, w, device="cuda")[None, None, :, None]
    ph = torch.rand(n, 1, 1, 4, device="cuda", generator=g) * 6.2831853
    base = 0.8 + 0.5 * torch.sin(9.0 * x + ph) * torch.cos(7.0 * y - ph)
    albedo = (0.5 + 0.4 * torch.sign(torch.sin(25.0 * x + ph) * torch.sin(21.0 * y + ph))).clamp(0.1, 0.9)
    clean = (base * albedo).clamp_min(0.0)
    noise = torch.exp(0.6 * torch.randn(n, h, w, 4, device="cuda", generator=g) - 0.18)
    fire = (torch.rand(n, h, w, 1, device="cuda", generator=g) < 1e-3).float() * 6.0
    rad = (clean * noise + fire).clamp(0.0, 10.0)
    nrm = torch.nn.functional.normalize(torch.sin(torch.cat([5 * x + 0 * y, 4 * y + 0 * x, 1 + x + y], 3) +
                                                  ph[..., :3]), dim=3)
    nrm = torch.cat([nrm, torch.ones_like(nrm[..., :1])], 3)
    wsum = torch.full((n, h, w, 4), 4.0, device="cuda") * (0.9 + 0.2 * torch.rand(n, h, w, 1, device="cuda",
                                                                                   generator=g))
    for t in (rad, albedo, clean):
        t[..., 3] = 1.0
    return rad.contiguous(), albedo.contiguous(), nrm.contiguous(), wsum.contiguous(), clean.contiguous()


def _params(seed):
    """Seeded He-normal network parameters in the network's parameter order."""
    rng = np.random.default_rng(seed)
    table = dn.layer_table()
    out = []
    for k, (cin, cout, _) in enumerate(table):
        sd = math.sqrt(2.0 / (9 * cin)) * (0.1 if k == len(table) - 1 else 1.0)
        out += [rng.standard_normal(cout * 9 * cin).astype(np.float32) * np.float32(sd),
                rng.uniform(-0.02, 0.02, cout).astype(np.float32)]
    return np.concatenate(out)


# ---- the cases ----------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _context():
    """A program keeps one context (a device and a stream) for all its work."""
    return ag.Context(0)


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    st = {"kind": kind, "ctx": ctx}
    if kind in ("box", "plugins", "sky", "mixed"):
        w, h, frames = case["width"], case["height"], case["frames"]
        if kind == "box":
            b, shot = scenes.box_scene(w, h, frames, case["depth"], seed=seed & 0xffffffff)
        elif kind == "plugins":
            b, shot = scenes.plugin_scene(w, h, frames, case["depth"], textured=case["textured"],
                                          opacity=case["opacity"], channels=("albedo", "normal", "depth"))
        elif kind == "sky":
            b, shot = scenes.sky_scene(w, h, frames, case["depth"], dusk=case["dusk"])
        else:
            b = _mixed_builder(case["spheres"], case["level"], seed)
            shot = _mixed_shot(b, case, w, h, frames, seed)
        shot.seed = seed & 0xffffffff
        film = ctx.create_film(w, h)
        st.update(scene=ctx.create_scene(b.desc()), shot=shot, film=film, out=_views(film))
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        b = _mixed_builder(case["spheres"], case["level"], seed)
        sides = [s for s in (64, 96, 160, 256, 384, 512) if s <= case["max_side"]]
        # every side and count in turn, so that each seed is the same amount of work
        st.update(scene=ctx.create_scene(b.desc()), shots=[], films=[], out=[])
        for k in range(case["shots"]):
            w = sides[k % len(sides)]
            h = w if k % 2 else w * 9 // 16
            spp = [s for s in (1, 4, 16) if s <= case["max_spp"]]
            z, a = float(rng.uniform(-0.4, 0.9)), float(rng.uniform(0.0, 6.2831853))
            r = math.sqrt(1.0 - z * z)
            st["shots"].append(_mixed_shot(b, case, w, h, spp[(k // 2) % len(spp)], (seed + k) & 0xffffffff,
                                           eye=(15.0 * r * math.cos(a), 15.0 * z, 15.0 * r * math.sin(a)),
                                           at=(0.0, 0.0, 0.0)))
            film = ctx.create_film(w, h)
            st["films"].append(film)
            st["out"].append(_views(film))
    elif kind == "load":
        b = _mixed_builder(case["spheres"], case["level"], seed)
        film = ctx.create_film(case["width"], case["height"])
        st.update(desc=b.desc(), film=film, out=_views(film),
                  shot=_mixed_shot(b, case, case["width"], case["height"], case["frames"], seed & 0xffffffff))
    elif kind == "denoise":
        w, h = case["width"], case["height"]
        film = ctx.create_film(w, h)
        ctx.sync()
        for k, img in zip((0, 1, 2, 8), _images(seed, 1, h, w)):
            film.tensor(k).copy_(img[0])
        align = 1 << (len(dn.DEFAULT_CHANNELS) - 1)
        den = dn.Denoiser(ctx, max_pixels=-(-h // align) * align * -(-w // align) * align)
        den.set_params(_params(seed))
        st.update(film=film, den=den, out=torch.empty(h, w, 4, device="cuda"))
    elif kind == "train":
        n, crop = case["batch"], case["crop"]
        den = dn.Denoiser(ctx, max_pixels=n * crop * crop, training=True)
        den.set_params(_params(seed))
        st.update(den=den, images=_images(seed, n, crop, crop))
    else:
        film = ctx.create_film(case["width"], case["height"])
        ctx.sync()
        film.tensor(0).copy_(_images(seed, 1, case["height"], case["width"])[0][0])
        post = ag.default_post({"none": A.TONEMAP_NONE, "gamma": A.TONEMAP_GAMMA, "filmic": A.TONEMAP_FILMIC,
                                "aces": A.TONEMAP_ACES, "pbrt": A.TONEMAP_PBRT}[case["operator"]])
        st.update(film=film, post=post)
    torch.cuda.synchronize()
    return st


def run(st):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "batch":
        ctx.render_batch(st["scene"], st["shots"], st["films"])
        return st["out"]
    if kind == "load":
        st["scene"] = ctx.create_scene(st["desc"])
        ctx.render(st["scene"], st["shot"], st["film"])
        return st["out"]
    if kind == "denoise":
        return st["den"].denoise(st["film"], out=st["out"])
    if kind == "train":
        with torch.cuda.stream(dn.ctx_stream(ctx)):
            rad, alb, nrm, wsum, target = st["images"]
            loss = st["den"].loss_grad(rad, alb, nrm, wsum, target)
            grads = st["den"].get_grads()
            st["den"].adam(1e-3)
        return {"loss": loss, "grads": grads}
    if kind == "tonemap":
        return ctx.tonemap(st["film"], 0, st["post"])
    ctx.render(st["scene"], st["shot"], st["film"])
    return st["out"]


# ---- what a pass cannot do without ----------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "denoise":
        align = 1 << (len(dn.DEFAULT_CHANNELS) - 1)
        h, w = (-(-case[k] // align) * align for k in ("height", "width"))
        return {"bytes": 5 * 16 * case["width"] * case["height"] + 2 * _params(0).size,
                "flops": dn.forward_flops(dn.DEFAULT_CHANNELS, h, w)}
    if kind == "train":
        p = case["batch"] * case["crop"] ** 2
        # forward, input gradient and weight gradient; Adam's four arrays read, three written
        return {"bytes": 5 * 16 * p + 4 * 8 * _params(0).size,
                "flops": 3.0 * case["batch"] * dn.forward_flops(dn.DEFAULT_CHANNELS, case["crop"], case["crop"])}
    if kind == "tonemap":
        return {"bytes": 2 * 16 * case["width"] * case["height"], "flops": 30 * case["width"] * case["height"]}
    if kind == "batch":
        sides = [s for s in (64, 96, 160, 256, 384, 512) if s <= case["max_side"]]
        spp = [s for s in (1, 4, 16) if s <= case["max_spp"]]
        shots = [(sides[k % len(sides)] * (sides[k % len(sides)] if k % 2 else sides[k % len(sides)] * 9 // 16),
                  spp[(k // 2) % len(spp)]) for k in range(case["shots"])]
        pixels, paths = sum(p for p, _ in shots), sum(p * s for p, s in shots)
    else:
        pixels = case["width"] * case["height"]
        paths = pixels * case["frames"]
    # rays a path traces on these scenes (camera, continuation, occlusion), and
    # the nodes of a balanced binary tree over the triangles that each must meet
    per_path = {"box": 2.0 * case["depth"], "plugins": 5.0, "sky": 4.0}.get(kind, 2.5)
    tris = {"box": 36, "plugins": 15000, "sky": 4000}.get(kind) or case["spheres"] * 20 * 4 ** case["level"] + 6
    flops = paths * per_path * (2 * 12 * math.log2(tris) + 2 * 40)
    scene = 0
    if kind == "load":
        scene = tris * (12 + 48) + tris / 2 * 64 + tris / 2 * 32  # indices and vertices in, triangles and nodes out
    elif kind in ("mixed", "batch"):
        scene = min(tris * 48, paths * per_path * 48)
    return {"bytes": pixels * 16 * len(FILM_IMAGES) + scene, "flops": flops}


# ---- 64-bit values ----------------------------------------------------------------
def _unet64(params, rad, alb, nrm, wsum):
    """The U-Net's head (3 channels) in 64 bits; images [n, h, w, 4] doubles."""
    F = torch.nn.functional
    ch, L = dn.DEFAULT_CHANNELS, len(dn.DEFAULT_CHANNELS)
    n, h, w, _ = rad.shape
    align = 1 << (L - 1)
    hp, wp = -(-h // align) * align, -(-w // align) * align
    x = torch.zeros(n, dn.IN_CHANNELS, hp, wp, dtype=torch.float64, device=rad.device)
    x[:, 0:3, :h, :w] = torch.log1p(rad[..., :3].clamp_min(0)).permute(0, 3, 1, 2)
    x[:, 3:6, :h, :w] = alb[..., :3].permute(0, 3, 1, 2)
    x[:, 6:9, :h, :w] = nrm[..., :3].permute(0, 3, 1, 2)
    x[:, 9, :h, :w] = torch.log2(1 + wsum[..., 0].clamp_min(0)) / 16
    at = [0, 0]

    def conv(t, relu=True):
        cin, cout, _ = dn.layer_table()[at[0]]
        k = cout * 9 * cin
        wgt = params[at[1]:at[1] + k].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        y = F.conv2d(t, wgt, params[at[1] + k:at[1] + k + cout], padding=1)
        at[0] += 1
        at[1] += k + cout
        return y.relu() if relu else y

    skips = []
    for l in range(L):
        x = conv(conv(x))
        if l < L - 1:
            skips.append(x)
            x = F.avg_pool2d(x, 2)
    for l in range(L - 2, -1, -1):
        x = conv(conv(torch.cat([F.interpolate(x, scale_factor=2, mode="nearest"), skips[l]], 1)))
    return conv(x, relu=False)[:, :3, :h, :w].permute(0, 2, 3, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("denoise", "train"):
        n, h, w = (1, case["height"], case["width"]) if kind == "denoise" else (case["batch"],) + (case["crop"],) * 2
        rad, alb, nrm, wsum, target = (t.double() for t in _images(seed, n, h, w))
        p = torch.from_numpy(_params(seed)).double().cuda().requires_grad_(kind == "train")
        log = torch.log1p(rad[..., :3].clamp_min(0))
        if kind == "denoise":
            with torch.no_grad():
                out = torch.expm1(_unet64(p, rad, alb, nrm, wsum) + log).clamp_min(0)
            return torch.cat([out, torch.ones_like(out[..., :1])], 3)[0]
        loss = (_unet64(p, rad, alb, nrm, wsum) + log - torch.log1p(target[..., :3].clamp_min(0))).abs().mean()
        loss.backward()
        return {"loss": float(loss), "grads": p.grad.cpu().numpy()}
    if kind == "tonemap":
        rad = _images(seed, 1, case["height"], case["width"])[0][0].double()
        c, op = rad[..., :3], case["operator"]
        if op == "gamma":
            c = (c / (c / 1.5 + 1)) ** (1 / 2.2)
        elif op == "filmic":
            c = (c - 0.004).clamp_min(0)
            c = (c * (c * 6.2 + 0.5)) / (c * (c * 6.2 + 1.7) + 0.06)
        elif op == "aces":
            c = ((c * (c * 2.51 + 0.03)) / (c * (c * 2.43 + 0.59) + 0.14)).clamp(0, 1) ** (1 / 2.2)
        elif op == "pbrt":
            c = torch.where(c < 0.0031308, 12.92 * c, 1.055 * c ** (1 / 2.4) - 0.055)
        return torch.cat([c, rad[..., 3:]], 2).cpu().numpy()
    return None  # a path-traced image has no value without the sample streams and the traversal themselves
