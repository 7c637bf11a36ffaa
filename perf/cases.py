"""The work whose speed is watched: ray queries, renders, batches of renders,
the adjoint and the post passes, through the package's public calls.

A case is a dict of plain values; its ``kind`` names the call:

* ``rays``     -- Model.rayHit / Model.rayHit_test over a device array of rays;
* ``render``   -- api.render of one scene into a Photo;
* ``batch``    -- Batch.update + Batch.render of several uneven renders;
* ``adjoint``  -- api.adjoint of a rendered Photo;
* ``display``  -- Photo.shade to a display image (gamma, FXAA);
* ``exports``  -- Photo.export_set, the images render_multiThread writes.

The scenes are the package's own generated ones (raym0nade_gb300.scenes). A
scene's geometry is the case's; the seed moves the camera a little and gives
the render's random streams, the rays, the loss gradient or the image.
"""
import functools
import math

import numpy as np
import torch

from raym0nade_gb300 import api, scenes


def listed():
    return [
        # picking and focus queries of an interactive program: a handful of rays, latency counts
        dict(name="pick", kind="rays", scene="terrain", tris=130050, n=1000, shadow=False),
        # the repository's traversal benchmark: incoherent closest-hit rays in a large soup
        dict(name="soup closest", kind="rays", scene="soup", tris=1000000, n=4000000, shadow=False),
        # visibility of a baked light: shadow rays over a terrain, an odd count
        dict(name="terrain shadow", kind="rays", scene="terrain", tris=2093058, n=1000003, shadow=True),
        # the preview while a camera moves: few pixels, few samples
        dict(name="preview", kind="render", scene="cornell", tris=36, width=160, height=90, spp=4, depth=8),
        # the Cornell box of the repository's benchmark
        dict(name="cornell", kind="render", scene="cornell", tris=36, width=256, height=256, spp=64, depth=8),
        # refraction and media, 16 times the paths behind glass
        dict(name="glass", kind="render", scene="glass", tris=36, width=250, height=250, spp=16, depth=16),
        # textures with mip chains, normal maps and alpha-tested cut-outs
        dict(name="textured", kind="render", scene="textured", tris=32, width=640, height=480, spp=32, depth=16),
        # the full-size frame: an open terrain under a sky at 1080p
        dict(name="terrain", kind="render", scene="terrain", tris=2093058, width=1920, height=1080, spp=64, depth=16),
        # a seeded set of uneven renders replayed per frame, soups and terrains mixed
        dict(name="batch", kind="batch", items=10, max_tris=300000, max_side=448, max_spp=96),
        # material gradients of an image loss
        dict(name="adjoint", kind="adjoint", scene="cornell16", tris=36, width=256, height=256, spp=32, depth=16),
        # every frame shown: composite, gamma and FXAA
        dict(name="display", kind="display", width=1280, height=720),
        # the images written after a final render, depth of field among them
        dict(name="exports", kind="exports", width=1920, height=1080, coc=6.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "render", "render", "render", "batch", "adjoint", "display", "exports"])
    if kind == "rays":
        return dict(kind=kind, scene=rng.choice(["soup", "terrain"]), tris=_log(rng, 1000, 2000000),
                    n=_log(rng, 100, 4000000), shadow=rng.random() < 0.5)
    if kind == "render":
        scene = rng.choice(["cornell", "glass", "textured", "terrain", "soup"])
        most = {"cornell": 600, "glass": 300, "textured": 800, "terrain": 1920, "soup": 800}[scene]
        width = _log(rng, 96, most)
        height = max(32, int(width * rng.uniform(0.5, 1.0)))
        tris = {"cornell": 36, "glass": 36, "textured": 32}.get(scene) or _log(rng, 1000, 2000000)
        return dict(kind=kind, scene=scene, tris=tris, width=width, height=height,
                    spp=_log(rng, 2, 16 if scene == "glass" else 64), depth=rng.randint(4, 16))
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(3, 12), max_tris=_log(rng, 10000, 300000),
                    max_side=_log(rng, 140, 448), max_spp=_log(rng, 16, 96))
    if kind == "adjoint":
        width = _log(rng, 32, 320)
        return dict(kind=kind, scene="cornell16", tris=36, width=width, height=max(24, int(width * rng.uniform(0.5, 1))),
                    spp=_log(rng, 4, 32), depth=rng.randint(4, 16))
    width = _log(rng, 120, 1920)
    height = max(64, int(width * rng.uniform(0.45, 0.8)))
    if kind == "display":
        return dict(kind=kind, width=width, height=height)
    return dict(kind=kind, width=width, height=height, coc=rng.choice([0.0, 2.0, 6.0]))


# ------------------------------------------------------------- scenes -----
@functools.lru_cache(maxsize=None)
def _sky(width, height):
    return scenes.sky_env(width, height)


@functools.lru_cache(maxsize=32)
def _scene(name, tris):
    if name == "cornell":
        return scenes.cornell()
    if name == "glass":
        return scenes.cornell_glass()
    if name == "textured":
        return scenes.textured_room()
    if name == "cornell16":
        return scenes.cornell16()
    if name == "soup":
        s = scenes.random_soup(tris, 1)
    else:
        s = scenes.heightfield(max(3, int(round(math.sqrt(tris / 2.0))) + 1), seed=3)
    s.env = _sky(1024, 512)
    return s


def _camera(case):
    w, h, spp, depth = case["width"], case["height"], case["spp"], case["depth"]
    if case["scene"] == "terrain":
        c = scenes.heightfield_camera(w, h, spp)
    elif case["scene"] == "textured":
        c = scenes.textured_camera(w, h, spp)
    elif case["scene"] == "soup":
        c = scenes.soup_camera(w, h, spp, depth)
    else:
        c = scenes.cornell_camera(w, h, spp)
    c.max_depth = depth
    return c


def _move(cam, seed):
    """A step of a moving camera: a small offset of its position."""
    r = np.random.default_rng(seed)
    cam.position = tuple(float(p) for p in np.asarray(cam.position) + r.uniform(-0.02, 0.02, 3))
    return cam


def _rays(case, seed):
    """Rays as a program has them on the device: incoherent ones inside the
    soup; over the terrain, picks straight at it or shadow rays from just
    above its surface toward the sky."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["n"]
    r = torch.empty((n, 8), device="cuda")
    d = torch.randn((n, 3), generator=g, device="cuda")
    r[:, 3] = 1e-4
    r[:, 7] = math.inf
    u = torch.rand((n, 3), generator=g, device="cuda")
    if case["scene"] == "soup":
        r[:, 0:3] = u
        if case["shadow"]:
            r[:, 7] = torch.rand(n, generator=g, device="cuda") * math.sqrt(3.0)
    else:
        s = _scene("terrain", case["tris"])
        side = int(round(math.sqrt(s.positions.shape[0])))
        height = torch.from_numpy(s.positions[:, 1].reshape(side, side).copy()).cuda()
        at = (u[:, [0, 2]] * (side - 1)).long()
        r[:, 0] = u[:, 0] * 200.0
        r[:, 2] = u[:, 2] * 200.0
        r[:, 1] = height[at[:, 1], at[:, 0]]
        if case["shadow"]:
            r[:, 1] += 0.2
            d[:, 1] = d[:, 1].abs() * 0.5 + 0.02
        else:
            r[:, 1] = 60.0
            d[:, 1] = -d[:, 1].abs() - 0.2
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    return r


# ------------------------------------------------------------- images -----
def _image(case, seed):
    """A rendered frame as the post passes meet it, made without a renderer:
    a floor and spheres under an empty sky (no hit: NaN positions), noisy
    radiance with fireflies. Returns the four radiance buffers, the G-buffer
    and the camera position."""
    w, h = case["width"], case["height"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rnd = lambda *k: torch.rand(k, generator=g, device="cuda")  # noqa: E731
    n = w * h
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    d = torch.stack([(x - w / 2) / w, (h / 2 - y) / w - 0.06, torch.ones_like(x, dtype=torch.float32)], -1).reshape(n, 3)
    d = d / d.norm(dim=1, keepdim=True)
    eye = torch.tensor([0.0, 1.2, 0.0], device="cuda")
    t = torch.where(d[:, 1] < -1e-3, -eye[1] / d[:, 1], math.inf)
    t = torch.where(t < 40.0, t, math.inf)
    normal = torch.tensor([0.0, 1.0, 0.0], device="cuda").repeat(n, 1)
    ident = torch.zeros(n, device="cuda")
    for k in range(12):
        c = torch.stack([rnd(1)[0] * 8 - 4, rnd(1)[0] * 1.5 + 0.3, rnd(1)[0] * 9 + 3])
        rad = rnd(1)[0] * 0.6 + 0.2
        oc = eye - c
        b = (d * oc).sum(1)
        q = b * b - (oc.dot(oc) - rad * rad)
        ts = torch.where(q > 0, -b - q.clamp_min(0).sqrt(), math.inf)
        near = (ts > 0) & (ts < t)
        t = torch.where(near, ts, t)
        normal = torch.where(near[:, None], (eye + ts[:, None] * d - c) / rad, normal)
        ident = torch.where(near, float(k + 1), ident)
    hit = torch.isfinite(t)
    palette, rough = rnd(13, 3) * 0.8 + 0.1, rnd(13) * 0.7 + 0.05
    metal = (rnd(13) < 0.3).float() * 0.8
    idx = ident.long()
    nan = torch.full((n, 3), math.nan, device="cuda")
    gb = torch.zeros((n, api.GBUFFER_FLOATS), device="cuda")
    gb[:, 0:3] = torch.where(hit[:, None], palette[idx], torch.zeros_like(nan))
    gb[:, 3:6] = torch.where(hit[:, None], torch.zeros_like(nan), 0.3 + 0.6 * d.abs())
    gb[:, 6:9] = torch.where(hit[:, None], eye + torch.where(hit, t, 0.0)[:, None] * d, nan)
    gb[:, 9:12] = torch.where(hit[:, None], normal, nan)
    gb[:, 12:15] = gb[:, 9:12]
    gb[:, 15], gb[:, 16] = torch.where(hit, rough[idx], 0.8), torch.where(hit, metal[idx], 0.0)
    gb[:, 17], gb[:, 18], gb[:, 19], gb[:, 20] = 1.0, 1.0, ident, 1.0
    shade = (normal * torch.tensor([0.4, 0.8, -0.45], device="cuda")).sum(1).clamp_min(0.05)
    rads = []
    for scale in (1.0, 0.3, 0.5, 0.2):
        noise = torch.exp(0.6 * torch.randn((n, 3), generator=g, device="cuda"))
        spark = 1.0 + 300.0 * (torch.rand((n, 1), generator=g, device="cuda") < 5e-4)
        c = torch.where(hit[:, None], scale * shade[:, None] * noise * spark, torch.zeros_like(nan))
        v = torch.where(hit, 0.4 * (c * c).sum(1) * torch.rand(n, generator=g, device="cuda"), torch.zeros(n, device="cuda"))
        rads.append(torch.cat([c, v[:, None]], 1).contiguous())
    return rads, gb, (0.0, 1.2, 0.0)


# --------------------------------------------------------------- calls -----
def prepare(case, seed):
    kind = case["kind"]
    if kind == "rays":
        return dict(case=case, model=api.Model(_scene(case["scene"], case["tris"])), rays=_rays(case, seed))
    if kind == "render":
        args = api.RenderArgs.from_camera(_move(_camera(case), seed), seed=seed)
        return dict(case=case, model=api.Model(_scene(case["scene"], case["tris"])), args=args,
                    photo=api.Photo(case["width"], case["height"]))
    if kind == "batch":
        # the repository's batch workload at a smaller size
        items, frames = [], []
        for i in range(case["items"]):
            r = np.random.default_rng(7 * 100003 + i)
            tris = int(math.exp(r.uniform(math.log(1e3), math.log(case["max_tris"]))))
            side = int(r.uniform(128, case["max_side"] + 1))
            spp = int(round(math.exp(r.uniform(math.log(8), math.log(case["max_spp"])))))
            c = dict(scene="soup" if r.random() < 0.5 else "terrain", tris=tris, width=side, height=side, spp=spp,
                     depth=int(r.integers(4, 17)))
            args = api.RenderArgs.from_camera(_camera(c), seed=7000 + i)
            items.append((api.Model(_scene(c["scene"], tris)), args, api.Photo(side, side)))
            frames.append(api.RenderArgs.from_camera(_move(_camera(c), seed + i), seed=seed + i))
        return dict(case=case, items=items, batch=api.Batch(items), frames=frames)
    if kind == "adjoint":
        args = api.RenderArgs.from_camera(_move(_camera(case), seed), seed=seed)
        model = api.Model(_scene(case["scene"], case["tris"]))
        photo = api.render(model, args)
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        # dL/dI of an L2 loss to a target near the image
        d = photo.shade(api.Full).reshape(-1, 3) * (torch.rand((case["width"] * case["height"], 3), generator=g,
                                                               device="cuda") - 0.3)
        return dict(case=case, model=model, args=args, photo=photo, d_image=d.contiguous())
    rads, gb, eye = _image(case, seed)
    photo = api.Photo(case["width"], case["height"])
    photo.Gbuffer = gb
    photo.focus, photo.CoC, photo.cameraPosition = 6.0, float(case.get("coc", 0.0)), eye
    photo.radiance_Dd, photo.radiance_Ds, photo.radiance_Id, photo.radiance_Is = (r.clone() for r in rads)
    return dict(case=case, photo=photo, raw=rads)


def run(state):
    kind = state["case"]["kind"]
    if kind == "rays":
        if state["case"]["shadow"]:
            return state["model"].rayHit_test(state["rays"])
        hits = state["model"].rayHit(state["rays"])
        return dict(face=hits[:, 0].view(torch.int32), t=hits[:, 1], bary=hits[:, 2:4])
    if kind == "render":
        p = api.render(state["model"], state["args"], state["photo"])
        return [p.radiance_Dd, p.radiance_Ds, p.radiance_Id, p.radiance_Is, p.Gbuffer]
    if kind == "batch":
        state["batch"].update(state["frames"])
        state["batch"].render()
        return [[p.radiance_Dd, p.radiance_Ds, p.radiance_Id, p.radiance_Is, p.Gbuffer]
                for _, _, p in state["items"]]
    if kind == "adjoint":
        return api.adjoint(state["model"], state["args"], state["photo"], state["d_image"])
    photo = state["photo"]
    if kind == "display":
        return photo.shade(api.Full | api.GAMMA | api.DoFXAA)
    # the clamp and the filter work in place: each frame starts from its render
    for buf, raw in zip((photo.radiance_Dd, photo.radiance_Ds, photo.radiance_Id, photo.radiance_Is), state["raw"]):
        buf.copy_(raw)
    images = photo.export_set()
    return dict(images=images, radiance=[photo.radiance_Dd, photo.radiance_Ds, photo.radiance_Id, photo.radiance_Is])


def work(case):
    """Bytes: inputs and outputs once, the scene once. Operations: the box and
    triangle tests and the shading that a path cannot do without (two boxes of
    18 operations a level, ten triangles of 45, 400 a shaded vertex)."""
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for i in range(case["items"]):
            r = np.random.default_rng(7 * 100003 + i)
            tris = int(math.exp(r.uniform(math.log(1e3), math.log(case["max_tris"]))))
            side = int(r.uniform(128, case["max_side"] + 1))
            spp = int(round(math.exp(r.uniform(math.log(8), math.log(case["max_spp"])))))
            w = work(dict(kind="render", tris=tris, width=side, height=side, spp=spp, depth=8, scene="soup"))
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "display":
        return dict(bytes=case["width"] * case["height"] * (4 * 16 + 24 + 12), flops=case["width"] * case["height"] * 120)
    if kind == "exports":
        images = 25 if case["coc"] > 1e-4 else 20
        n = case["width"] * case["height"]
        # the filter's 5 passes x 25 taps on four buffers and the images' own arithmetic
        return dict(bytes=n * (8 * 16 + 84 + 12 * images), flops=n * (5 * 25 * 4 * 30 + images * 120))
    tris = case["tris"]
    levels = max(1.0, math.log2(max(2, tris) / 8.0))
    ray = levels * 2 * 18 + 10 * 45
    scene = tris * (48 + 64 / 8)
    if kind == "rays":
        return dict(bytes=case["n"] * (32 + (1 if case["shadow"] else 16)) + scene, flops=case["n"] * ray)
    n = case["width"] * case["height"]
    paths = n * case["spp"]
    rays = paths * (1.0 if kind == "render" else 1.5)
    return dict(bytes=n * (4 * 16 + 84 + 12) + scene, flops=rays * (ray + 400))


# -------------------------------------------------------- in 64 bits -----
def exact(case, seed):
    kind = case["kind"]
    if kind == "rays" and not case["shadow"] and case["n"] * case["tris"] <= 2e8:
        return dict(face=None, t=_closest(_scene(case["scene"], case["tris"]), _rays(case, seed)), bary=None)
    if kind == "display":
        rads, gb, _ = _image(case, seed)
        return _fxaa(_gamma(_shade(rads, gb, "full")), case["width"], case["height"])
    if kind == "exports":
        return _exports(case, seed)
    return None  # Monte Carlo paths: a rounding moves a path's branches


def _closest(scene, rays):
    p = torch.from_numpy(scene.positions).cuda().double()[torch.from_numpy(scene.indices).cuda().long()]
    v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    r = rays.double()
    out = []
    step = max(1, int(2e6) // v0.shape[0])
    for k in range(0, r.shape[0], step):
        o, d = r[k:k + step, None, 0:3], r[k:k + step, None, 4:7]
        h = torch.cross(d.expand(-1, e2.shape[0], -1), e2[None].expand(d.shape[0], -1, -1), dim=-1)
        a = (e1 * h).sum(-1)
        s = o - v0
        u = (s * h).sum(-1) / a
        q = torch.cross(s, e1[None].expand(s.shape[0], -1, -1), dim=-1)
        v = (d * q).sum(-1) / a
        t = (e2 * q).sum(-1) / a
        ok = (a.abs() / e1.norm(dim=1) >= 1e-4) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-4)
        out.append(torch.where(ok, t, math.inf).min(dim=1).values)
    return torch.cat(out)


_LUM = (0.3, 0.6, 0.1)


def _lum(c):
    return c[..., 0] * _LUM[0] + c[..., 1] * _LUM[1] + c[..., 2] * _LUM[2]


def _shade(rads, gb, what):
    """Photo::shade of one export: base colour, a normal, one buffer, or all."""
    gb = gb.double()
    if what == "base":
        return gb[:, 0:3]
    if what in ("shape", "surface"):
        k = 9 if what == "shape" else 12
        return (gb[:, k:k + 3] + 1.0) / 2.0
    dd, ds, di, si = (r.double()[:, 0:3] for r in rads)
    if what == "full":
        return gb[:, 0:3] * (dd + di) + ds + si + gb[:, 3:6]
    return {"Dd": dd, "Ds": ds, "Id": di, "Is": si}[what]


def _gamma(p):
    p = torch.where(p < 0.0, 0.0, p)  # a NaN channel stays
    c = _lum(p)[:, None]
    p = torch.where(c > 0.75, p / c * (torch.tanh(3.0 * (c - 0.75)) / 3.0 + 0.75), p)
    p = torch.where(p > 1.0, 1.0, p)
    return p ** (1.0 / 2.2)


def _at(img, dy, dx):
    """img (h, w, k) read at (y + dy, x + dx) and where that lies inside."""
    h, w = img.shape[:2]
    y = torch.arange(h, device=img.device) + dy
    x = torch.arange(w, device=img.device) + dx
    inside = ((y >= 0) & (y < h))[:, None] & ((x >= 0) & (x < w))[None, :]
    return img[y.clamp(0, h - 1)][:, x.clamp(0, w - 1)], inside


def _fxaa(rgb, w, h):
    img = rgb.reshape(h, w, 3)
    lum = _lum(img)[..., None]

    def near(dy, dx):
        v, ok = _at(lum, dy, dx)
        return torch.where(ok, v[..., 0], lum[..., 0])

    M, N, S, E, W = lum[..., 0], near(-1, 0), near(1, 0), near(0, 1), near(0, -1)
    lo = torch.minimum(torch.minimum(N, S), torch.minimum(E, W))
    hi = torch.maximum(torch.maximum(N, S), torch.maximum(E, W))
    rng = hi - lo
    keep = rng < torch.maximum(torch.full_like(hi, 0.0312), hi * 0.125)
    NW, NE, SW, SE = near(-1, -1), near(-1, 1), near(1, -1), near(1, 1)
    eh = ((NW + W + SW) - (NE + E + SE)).abs() / 3.0
    ev = ((NW + N + NE) - (SW + S + SE)).abs() / 3.0
    horiz = eh >= ev
    step = torch.where(horiz, 1.0 / w, 1.0 / h)
    g = (torch.where(horiz, eh, ev) / rng).clamp(-2.0, 2.0)
    ys, xs = torch.meshgrid(torch.arange(h, device=img.device), torch.arange(w, device=img.device), indexing="ij")
    best, by, bx = torch.zeros_like(M), ys.clone(), xs.clone()
    for i in range(12):
        off = torch.nan_to_num(g * step * (i + 1))
        sx, sy = xs / w + torch.where(horiz, 0.0, off), ys / h + torch.where(horiz, off, 0.0)
        ok = (sx >= 0) & (sx <= 1) & (sy >= 0) & (sy <= 1)
        ix, iy = (sx * w + 1e-9).long().clamp(0, w - 1), (sy * h + 1e-9).long().clamp(0, h - 1)
        d = (M[iy, ix] - M).abs()
        take = ok & (d > best)
        best, by, bx = torch.where(take, d, best), torch.where(take, iy, by), torch.where(take, ix, bx)
    sub = (((N + S - 2 * M).abs() * 2 + (E + W - 2 * M).abs()) * 0.25).clamp(max=1.0)
    a = (sub * 0.75)[..., None]
    return torch.where(keep[..., None], img, img * (1 - a) + img[by, bx] * a)


def _bloom(rgb, w, h):
    img = rgb.reshape(h, w, 3)
    c = _lum(img)[..., None]
    b = torch.where(c < 1.0, 0.0, (img / c ** 0.65 - 1.0).clamp_min(0.0))
    k5 = (0.0625, 0.25, 0.375, 0.25, 0.0625)
    for step in (1, 2, 4, 8, 16):
        out = torch.zeros_like(b)
        for i in range(5):
            for j in range(5):
                v, ok = _at(b, (i - 2) * step, (j - 2) * step)
                out = out + torch.where(ok[..., None], v, 0.0) * k5[i] * k5[j]
        b = out
        img = img + b / 6.0
    return img.reshape(-1, 3)


def _spatial_clamp(rad, w, h):
    k7 = (0.03125, 0.109375, 0.21875, 0.28125, 0.21875, 0.109375, 0.03125)
    l = _lum(rad).reshape(h, w, 1)
    for axis in (1, 0):
        out = torch.zeros_like(l) if axis == 1 else out
        src, acc = (l, torch.zeros_like(l)) if axis == 1 else (out, torch.zeros_like(l))
        for i in range(7):
            v, ok = _at(src, 0 if axis == 1 else i - 3, i - 3 if axis == 1 else 0)
            acc = acc + torch.where(ok[..., None], v, 0.0) * k7[i]
        out = acc
    bl = (out - k7[3] * k7[3] * l).reshape(-1)
    l = l.reshape(-1)
    s = torch.where(l > 36.0 * bl, bl / (l + 1e-4) / (1.0 - k7[3] * k7[3]), 1.0)
    return torch.cat([rad[:, 0:3] * s[:, None], rad[:, 3:4]], 1)


def _filter(rads, gb, w, h):
    """Photo::filter: the variance's 3x3 pass, then five a-trous passes."""
    gb = gb.double().reshape(h, w, -1)
    pos, shape_n, surf_n = gb[..., 6:9], gb[..., 9:12], gb[..., 12:15]
    rough, metal, opac = gb[..., 15], gb[..., 16], gb[..., 17]
    hit = torch.isfinite(pos).any(-1)
    cur = []
    for r in rads:
        img = r.reshape(h, w, 4)
        E, E2, V = torch.zeros_like(img[..., 0:3]), torch.zeros_like(img[..., 0]), torch.zeros_like(img[..., 0])
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                q, ok = _at(img, dy, dx)
                wt = torch.where(ok, (0.5 if dx == 0 else 0.25) * (0.5 if dy == 0 else 0.25), 0.0)
                E, E2, V = E + q[..., 0:3] * wt[..., None], E2 + (q[..., 0:3] ** 2).sum(-1) * wt, V + q[..., 3] * wt
        cur.append(torch.cat([img[..., 0:3], (V + E2 - (E * E).sum(-1))[..., None]], -1))
    k5 = (0.0625, 0.25, 0.375, 0.25, 0.0625)
    for step in (1, 2, 4, 8, 16):
        acc = [[torch.zeros_like(pos), torch.zeros_like(rough), torch.zeros_like(rough)] for _ in cur]
        for i in range(5):
            for j in range(5):
                dy, dx = (i - 2) * step, (j - 2) * step
                gq, ok = _at(gb, dy, dx)
                centre = i == 2 and j == 2
                if not centre:
                    wn = (surf_n * gq[..., 12:15]).sum(-1).clamp_min(0.0) ** 1024
                    e = gq[..., 6:9] - pos
                    st = (shape_n * (e / e.norm(dim=-1, keepdim=True))).sum(-1).abs()
                    tt = st / ((1.0 - st * st).sqrt() + 1e-4)
                    md = ((metal - gq[..., 16]) ** 2 + (opac - gq[..., 17]) ** 2).sqrt()
                    ok2 = ok & torch.isfinite(gq[..., 6:9]).any(-1) & ~(wn < 1e-6)
                for b, img in enumerate(cur):
                    q, _ = _at(img, dy, dx)
                    wt = torch.full_like(rough, k5[i] * k5[j])
                    if not centre:
                        rd = (img[..., 0:3] - q[..., 0:3]).norm(dim=-1) / (img[..., 3].sqrt() + 1e-2)
                        k = -tt - rd - md
                        we = wn * torch.exp(k)
                        if b % 2 == 1:
                            we = we * rough.clamp_min(4e-2)
                        wt = wt * torch.where(ok2 & ~(k < -7.5) & torch.isfinite(we), we, 0.0)
                        q = torch.where(ok[..., None], q, 0.0)
                    acc[b][0] = acc[b][0] + q[..., 0:3] * wt[..., None]
                    acc[b][1] = acc[b][1] + q[..., 3] * wt * wt
                    acc[b][2] = acc[b][2] + wt
        cur = [torch.where(hit[..., None], torch.cat([c / ws[..., None], (v / (ws * ws))[..., None]], -1), 0.0)
               for c, v, ws in acc]
    return [c.reshape(-1, 4) for c in cur]


def _exports(case, seed):
    """The exports without FXAA and depth of field, and the filtered buffers.
    FXAA's and the depth-of-field blur's choices turn on roundings."""
    w, h = case["width"], case["height"]
    rads, gb, _ = _image(case, seed)
    rads = [r.double() for r in rads]
    im = lambda p: _gamma(p).reshape(h, w, 3)  # noqa: E731
    out = dict(DiffuseColor=im(_shade(rads, gb, "base")), DiffuseColor_FXAA=None,
               shapeNormal=im(_shade(rads, gb, "shape")), surfaceNormal=im(_shade(rads, gb, "surface")))
    rads = [_spatial_clamp(r, w, h) for r in rads]
    for stage in ("", "_Filter"):
        if stage:
            rads = _filter(rads, gb, w, h)
        for tag, key in (("Direct_Diffuse", "Dd"), ("Direct_Specular", "Ds"), ("Indirect_Diffuse", "Id"),
                         ("Indirect_Specular", "Is")):
            out[tag + stage] = im(_shade(rads, gb, key))
        name = "Filter" if stage else "Raw"
        full = _shade(rads, gb, "full")
        out[name], out[name + "_Bloom"] = im(full), im(_bloom(full, w, h))
        out[name + "_FXAA"] = out[name + "_Bloom_FXAA"] = None
    if case["coc"] > 1e-4:
        for tag in ("BaseColor_DepthFieldBlur", "Filter_DepthFieldBlur", "Filter_DepthFieldBlur_Bloom",
                    "Filter_DepthFieldBlur_FXAA", "Filter_DepthFieldBlur_Bloom_FXAA"):
            out[tag] = None
    return dict(images=out, radiance=rads)
