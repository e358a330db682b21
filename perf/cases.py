"""Performance cases of the foveated HTGS renderer: the frames its users render.

Every case is one call through a public entry point on a seeded synthetic scene with the
benchmark distributions (positions N(0,1)^3 rescaled to a 4-unit box, log-scales N(-4.5, 0.5),
random unit quaternions, opacities sigmoid(N(0, 1.5)), SH DC N(0, 0.3), higher bands
N(0, 0.05)) seen by pinhole cameras that look at the origin.  The entry points:

* `render` / `benchmark` / `stereo`: the drop-in blocking calls of `FoveatedHTGSRasterizer`
  (IEEE arithmetic for `render`, fast math for the other two; fresh images per call);
* `frame`: `Renderer.render(sync=False)` into images the program keeps;
* `graph`: a captured `FrameGraph`, replayed;
* `display`: a headset frame: tile masks from a lens map on the device, the stereo frame, the
  8-bit side-by-side image;
* `served`: a burst of stereo requests through the request `Server`.

`exact` restates the frame in 64 bits with plain torch operations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import foveatedhtgscudabackend_b200 as fhtgs
from foveatedhtgscudabackend_b200 import display, scene

TILE = 16
FOVEA_TILES, BLEND_TILES, BLEND_WIDTH_PX = 24, 15, 125  # the reference layout's radii
MIN_ALPHA, MIN_ALPHA_CORE, MAX_CUTOFF_SQ, MIN_T = 1.0 / 255.0, 1.0 / 20.0, 11.0825270903, 1e-4
RINGS = (0.15, 0.4)
N_REQUESTS = 4          # requests of a served burst
EXACT_GAUSSIANS = 150_000  # largest Gaussians x views that `exact` evaluates in seconds

DEFAULTS = dict(api="frame", n=100_000, sh=3, views=1, width=1280, height=720, K=8, foveation="reference",
                storage="fp32", aaa=False, blur=False, background="none", chw=True, distance=6.0)


def _case(name: str | None = None, **kw) -> dict:
    case = dict(DEFAULTS, **kw)
    return case if name is None else dict(case, name=name)


def listed() -> list[dict]:
    return [
        # a thumbnail or a probe view: the smallest call, latency and launches
        _case("tiny_render", api="render", n=2_000, sh=1, width=320, height=240, K=4),
        # the plain view: one 1280x720 image of a small SH0 scene without foveation, replayed
        _case("plain_graph", api="graph", n=100_000, sh=0, K=4, foveation="none"),
        # the reference's benchmark call on a desktop view, ragged size, channels last
        _case("benchmark_ragged", api="benchmark", n=60_000, sh=2, width=1003, height=757, K=8, chw=False),
        # the quality options together: IEEE arithmetic, anti-aliasing, blurred periphery, K = 16
        _case("render_quality", api="render", n=300_000, sh=3, width=1920, height=1080, K=16, aaa=True, blur=True,
              background="sh"),
        # the headline headset frame: 1M Gaussians, two 2064x2208 eyes, reference foveation
        _case("stereo_headline", api="frame", n=1_000_000, views=2, width=2064, height=2208),
        # the same class of frame through the blocking drop-in call
        _case("stereo_dropin", api="stereo", n=500_000, views=2, width=1440, height=1584),
        # ring foveation of a large scene in reduced-precision storage
        _case("rings_half", api="frame", n=6_000_000, views=2, width=2064, height=2208, foveation="rings",
              storage="half"),
        # a close view: long lists and large footprints, deep K-buffer
        _case("close_k32", api="frame", n=150_000, sh=1, width=1280, height=720, K=32, distance=3.0),
        # many cameras of one scene in one captured frame
        _case("batched_graph", api="graph", n=1_000_000, views=12, width=1920, height=1080),
        # a headset frame with lens masks and the 8-bit image for the display
        _case("display_lens", api="display", n=250_000, views=2, width=1440, height=1584, foveation="rings"),
        # concurrent stereo requests on one resident scene
        _case("served_burst", api="served", n=500_000, views=2, width=1440, height=1584),
    ]


def draw(rng) -> dict:
    api = rng.choice(["render", "benchmark", "stereo", "frame", "frame", "graph", "graph", "display", "served"])
    n = int(round(math.exp(rng.uniform(math.log(2_000), math.log(1_500_000)))))
    K = rng.choice([1, 2, 4, 8, 8, 8, 16, 32])
    if rng.random() < 0.4:
        width, height = rng.choice([(640, 480), (1280, 720), (1920, 1080), (1440, 1584), (2064, 2208)])
    else:
        width = int(round(math.exp(rng.uniform(math.log(200), math.log(2064)))))
        height = int(round(math.exp(rng.uniform(math.log(200), math.log(2208)))))
    views = 2 if api in ("stereo", "display", "served") else 1
    if api in ("frame", "graph"):
        views = rng.choice([1, 2, 2, 3, 6])
    # a frame costs no more than the largest listed one, also a small image, whose lists are long
    n = min(n, 2_500_000 // (views * (N_REQUESTS if api == "served" else 1)), 250_000 if K > 8 else n)
    dropin = api in ("render", "benchmark", "stereo")
    foveation = "reference" if dropin else rng.choice(["reference", "reference", "rings", "none"])
    return _case(api=api, n=n, sh=rng.choice([0, 1, 2, 3, 3]), views=views, width=width, height=height, K=K,
                 foveation=foveation, storage="fp32" if dropin else rng.choice(["fp32", "fp32", "half"]),
                 aaa=rng.random() < 0.2, blur=foveation == "reference" and rng.random() < 0.25,
                 background=rng.choice(["none", "none", "sh"]), chw=rng.random() < 0.7,
                 distance=round(rng.uniform(3.5, 8.0), 2))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _gaussians(case: dict, seed: int) -> tuple[torch.Tensor, ...]:
    """(positions, scales, rotations, opacities, sh_0, sh_rest) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, rest = case["n"], (case["sh"] + 1) ** 2 - 1

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    pos = normal(n, 3)
    pos = pos * (2.0 / pos.abs().max())
    scales = torch.exp(normal(n, 3) * 0.5 - 4.5)
    rot = normal(n, 4)
    rot = rot / rot.norm(dim=1, keepdim=True)
    opacities = torch.sigmoid(normal(n, 1) * 1.5)
    out = (pos, scales, rot, opacities, normal(n, 1, 3) * 0.3, normal(n, rest, 3) * 0.05)
    return fhtgs.torch_scene.to_half_storage(*out) if case["storage"] == "half" else out


def _views(case: dict, seed: int, request: int = 0) -> list[scene.View]:
    """The case's cameras: a stereo pair for two views, else cameras around the scene."""
    rng = np.random.default_rng(1000 * seed + request)
    w, h = case["width"], case["height"]
    pairs = (case["views"] + 1) // 2
    out = []
    for _ in range(pairs):
        a = rng.uniform(0.0, 2.0 * math.pi)
        d = np.array([math.sin(a), rng.uniform(-0.3, 0.3), -math.cos(a)])
        position = tuple(case["distance"] * d / np.linalg.norm(d))
        gaze = tuple(np.clip(rng.normal(0.0, 0.05, size=2), -0.9, 0.9))
        for eye in (-0.0315, 0.0315):
            out.append(scene.make_view(w, h, position=position, eye_offset=eye, gaze_ndc=gaze))
    return out[:case["views"]]


def _background(case: dict, seed: int):
    return scene.sh_background(seed) if case["background"] == "sh" else None


def _lens(case: dict) -> np.ndarray:
    gw, gh = -(-case["width"] // TILE), -(-case["height"] // TILE)
    return scene.lens_visibility(gw, gh)


def prepare(case: dict, seed: int):
    g = _gaussians(case, seed)
    bg = _background(case, seed)
    model = fhtgs.BackgroundModel.SH if bg is not None else fhtgs.BackgroundModel.NONE
    state = dict(case=case, g=g)
    if case["api"] == "served":
        server = fhtgs.Server(device=g[0].device)
        state["server"] = server
        state["scene"] = server.add_scene(
            *g, K=case["K"], active_sh_bases=(case["sh"] + 1) ** 2, to_chw=case["chw"], blur_periphery=case["blur"],
            aaa_mode=case["aaa"], background=model,
            background_data=None if bg is None else torch.from_numpy(bg).cuda(), foveation=case["foveation"],
            rings=RINGS)
        state["requests"] = [_views(case, seed, r) for r in range(N_REQUESTS)]
        state["images"] = [[_image(case) for _ in eyes] for eyes in state["requests"]]
        return state
    state["settings"] = [fhtgs.settings_from_view(v, K=case["K"], active_sh_bases=(case["sh"] + 1) ** 2,
                                                  background=model, background_data=bg)
                         for v in _views(case, seed)]
    state["options"] = (case["chw"], case["blur"], case["aaa"])
    if case["api"] in ("render", "benchmark", "stereo"):
        state["rasterizer"] = fhtgs.FoveatedHTGSRasterizer()
        return state
    renderer = fhtgs.Renderer(g[0].device)
    renderer.set_foveation(case["foveation"], *RINGS)
    state["renderer"] = renderer
    state["images"] = [_image(case) for _ in range(case["views"])]
    if case["api"] == "graph":
        state["graph"] = renderer.capture(*g, state["settings"], *state["options"], images=state["images"])
        return state
    if case["api"] == "display":
        state["lens"] = torch.from_numpy(_lens(case)).cuda()
        state["packed"] = torch.empty((case["height"], case["views"] * case["width"], 4), dtype=torch.uint8,
                                      device="cuda")
    # the program's first frame is a blocking one: it sizes the instance capacity
    renderer.render(*g, state["settings"], *state["options"], images=state["images"])
    return state


def _image(case: dict) -> torch.Tensor:
    h, w = case["height"], case["width"]
    return torch.zeros((3, h, w) if case["chw"] else (h, w, 3), device="cuda")


def run(state):
    case, g = state["case"], state["g"]
    api = case["api"]
    if api == "served":
        server = state["server"]
        for eyes, images in zip(state["requests"], state["images"]):
            server.submit(state["scene"], eyes, images)
        done = 0
        while done < len(state["requests"]):
            for c in server.poll(wait_ms=100):
                if not c.ok:
                    raise RuntimeError(c.message)
                done += 1
        return state["images"]
    if api == "render":
        return state["rasterizer"].render(*g, state["settings"][0], *state["options"])
    if api == "benchmark":
        return state["rasterizer"].benchmark(*g, state["settings"][0], *state["options"])
    if api == "stereo":
        return state["rasterizer"].render_stereo(*g, *state["settings"], *state["options"])
    if api == "graph":
        return state["graph"].launch()
    settings = state["settings"]
    if api == "display":
        words, sat, fovea = display.build_tile_masks(case["width"], case["height"], state["lens"])
        settings = [s._replace(visibility_mask=words, visibility_mask_area_table=sat, fovea_mask_area_table=fovea)
                    for s in settings]
    images = state["renderer"].render(*g, settings, *state["options"], images=state["images"], sync=False)
    if api == "display":
        return images, display.pack_display(images, to_chw=case["chw"], out=state["packed"])
    return images


# ------------------------------------------------------------------------------------------
# work a frame cannot do without
# ------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Bytes: every attribute read once, every image written once.  Flops: 45 for each pair of a
    Gaussian and a sample inside its cutoff ellipse (plane, distance, exponential, accumulation);
    the pairs from 4,096 Gaussians of the distributions (seed 0)."""
    gen = torch.Generator().manual_seed(0)
    m = 4096
    pos = torch.randn(m, 3, generator=gen)
    pos = pos * (2.0 / 4.6)  # the largest of 3 N normal values, nearly independent of N
    sigma = torch.exp(torch.randn(m, 2, generator=gen).mean(1) * 0.5 - 4.5)
    opacity = torch.sigmoid(torch.randn(m, generator=gen) * 1.5)
    w, h = case["width"], case["height"]
    focal = 0.5 * h / math.tan(math.radians(30.0))
    z = pos[:, 2] + case["distance"]
    x, y = focal * pos[:, 0] / z, focal * pos[:, 1] / z  # pixels from the image centre
    area = math.pi * (focal * sigma / z) ** 2 * (2.0 * torch.log(255.0 * opacity)).clamp(min=0.0, max=MAX_CUTOFF_SQ)
    inside = (x.abs() < 0.5 * w) & (y.abs() < 0.5 * h)
    density = torch.ones(m)
    if case["foveation"] == "reference":
        density = torch.where(x * x + y * y < (FOVEA_TILES * TILE) ** 2, 1.0, 0.25)
    elif case["foveation"] == "rings":
        r2 = (2.0 * x / w) ** 2 + (2.0 * y / h) ** 2
        density = torch.where(r2 < RINGS[0] ** 2, 1.0, torch.where(r2 < RINGS[1] ** 2, 0.25, 0.0625))
    frames = case["views"] * (N_REQUESTS if case["api"] == "served" else 1)
    pairs = frames * case["n"] * float((area * inside * density).mean())
    values = 3 * (case["sh"] + 1) ** 2
    per_gaussian = 12 + 2 * (8 + values) if case["storage"] == "half" else 4 * (11 + values)
    pixel_bytes = 12 + (4 if case["api"] == "display" else 0)
    return {"bytes": case["n"] * per_gaussian + frames * w * h * pixel_bytes, "flops": 45.0 * pairs}


# ------------------------------------------------------------------------------------------
# the frame in 64 bits
# ------------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    requests = N_REQUESTS if case["api"] == "served" else 1
    if case["n"] * case["views"] * requests > EXACT_GAUSSIANS or (case["aaa"] and case["distance"] < 5.0):
        return None  # too many steps; or cameras among Gaussians, where anti-aliasing bounds them otherwise
    g = [t.double() for t in _gaussians(case, seed)]
    bg = _background(case, seed)
    bg = None if bg is None else torch.from_numpy(bg).cuda().double()
    images = [[_exact_view(case, g, v, bg) for v in _views(case, seed, r)] for r in range(requests)]
    if not case["chw"]:
        images = [[im.permute(1, 2, 0).contiguous() for im in eyes] for eyes in images]
    if case["api"] == "served":
        return images
    images = images[0]
    if case["api"] == "display":
        return images, None
    return images[0] if case["api"] in ("render", "benchmark") else images


def _sh_sum(c: torch.Tensor, d: torch.Tensor) -> torch.Tensor:
    """0.5 + the real SH expansion (degree <= 3) of coefficients c [..., B, 3] along d [..., 3]."""
    x, y, z = d.unbind(-1)
    xx, yy, zz = x * x, y * y, z * z
    basis = [torch.full_like(x, 0.28209479177387814), -0.48860251190291987 * y, 0.48860251190291987 * z,
             -0.48860251190291987 * x, 1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
             0.94617469575755997 * zz - 0.31539156525251999, -1.0925484305920792 * x * z,
             0.54627421529603959 * (xx - yy), y * (0.59004358992664352 * yy - 1.7701307697799304 * xx),
             2.8906114426405538 * x * y * z, y * (0.45704579946446572 - 2.2852289973223288 * zz),
             z * (1.865881662950577 * zz - 1.1195289977703462), x * (0.45704579946446572 - 2.2852289973223288 * zz),
             1.4453057213202769 * z * (xx - yy), x * (1.7701307697799304 * yy - 0.59004358992664352 * xx)]
    out = 0.5
    for k in range(c.shape[-2]):
        out = out + basis[k].unsqueeze(-1) * c[..., k, :]
    return out


def _tensor(a) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


def _project(case, g, v):
    """Visible Gaussians of one view: index order, records (P1, P2, P4, rgb, opacity), tile bounds."""
    pos, scale, q, opacity, sh0, rest = g
    opacity = opacity.reshape(-1)
    M, VPM, cam = _tensor(v.M), _tensor(v.VPM), _tensor(v.cam_position)
    z = pos @ M[2, :3] + M[2, 3]
    keep = (z >= v.near_plane) & (z <= v.far_plane)
    r, x, y, w = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + w * w), 2 * (x * y - r * w), 2 * (r * y + x * w),
                     2 * (x * y + r * w), 1 - 2 * (x * x + w * w), 2 * (y * w - r * x),
                     2 * (x * w - r * y), 2 * (y * w + r * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    if case["aaa"]:
        var = scale * scale + (0.3 * (z / max(v.focal_x, v.focal_y)) ** 2).unsqueeze(1)
        d = pos - cam
        d = d / d.norm(dim=1, keepdim=True)
        d2 = torch.einsum("nij,ni->nj", R, d) ** 2

        def det(s):
            return (d2 * torch.stack([s[:, 1] * s[:, 2], s[:, 2] * s[:, 0], s[:, 0] * s[:, 1]], 1)).sum(1)

        opacity = opacity * torch.sqrt((det(scale * scale) / det(var)).clamp(0.0, 1.0))
        scale = torch.sqrt(var)
        keep = opacity >= MIN_ALPHA  # no depth test in this mode
    cutoff = 2.0 * torch.log(opacity * 255.0)
    T = torch.cat([R * scale.unsqueeze(1), pos.unsqueeze(2)], 2)  # columns u, v, w, centre
    P = torch.einsum("rk,nkc->nrc", VPM[:, :3], T)
    P[:, :, 3] += VPM[:, 3]
    t = torch.stack([cutoff, cutoff, cutoff, -torch.ones_like(cutoff)], 1)
    s = (t * P[:, 3] ** 2).sum(1)
    keep &= s != 0
    f = t / s.unsqueeze(1)

    def extent(row):
        c = (f * P[:, row] * P[:, 3]).sum(1)
        return c, torch.sqrt((c * c - (f * P[:, row] ** 2).sum(1)).clamp(min=0.0))

    (cx, ex), (cy, ey), (cz, ez) = extent(0), extent(1), extent(2)
    if not case["aaa"]:
        keep &= (cz - ez >= -1.0) & (cz + ez <= 1.0)
    gw, gh = v.grid_large

    def tiles(c, e, n):
        return (((c - e + 0.5) / TILE).floor().clamp(0, n), ((c + e + 0.5) / TILE).ceil().clamp(0, n))

    b = torch.stack([*tiles(cx, ex, gw), *tiles(cy, ey, gh)], 1)
    keep &= (b[:, 1] > b[:, 0]) & (b[:, 3] > b[:, 2])
    i = keep.nonzero().squeeze(1)
    d = pos[i] - cam
    rgb = _sh_sum(torch.cat([sh0.reshape(-1, 1, 3), rest], 1)[i], d / d.norm(dim=1, keepdim=True))
    return P[i, 0], P[i, 1], P[i, 3], rgb, opacity[i], b[i].long()


def _tile_strides(case, v) -> tuple[torch.Tensor, torch.Tensor]:
    """Per tile [gh, gw]: sample stride (0: masked) and whether it is a blended tile."""
    gw, gh = v.grid_large
    ty, tx = torch.meshgrid(torch.arange(gh, device="cuda").double(), torch.arange(gw, device="cuda").double(),
                            indexing="ij")
    gaze = _tensor(v.gaze_position)
    blended = torch.zeros(gh, gw, dtype=torch.bool, device="cuda")
    stride = torch.ones(gh, gw, dtype=torch.long, device="cuda")
    if case["foveation"] == "reference":
        g = ((gaze.long() + TILE // 2) // TILE).double()
        d2 = (tx + 0.5 - g[0]) ** 2 + (ty + 0.5 - g[1]) ** 2
        stride[d2 >= FOVEA_TILES ** 2] = 2
        blended = (d2 < FOVEA_TILES ** 2) & (d2 >= BLEND_TILES ** 2)
    elif case["foveation"] == "rings":
        r2 = (((tx * TILE + TILE / 2) - gaze[0]) / (0.5 * v.width)) ** 2 + \
             (((ty * TILE + TILE / 2) - gaze[1]) / (0.5 * v.height)) ** 2
        stride[r2 >= RINGS[0] ** 2] = 2
        stride[r2 >= RINGS[1] ** 2] = 4
    if case["api"] == "display":
        stride[~torch.from_numpy(_lens(case)).cuda()] = 0
    return stride, blended


def _exact_view(case, g, v, bg):
    P1, P2, P4, rgb, opacity, b = _project(case, g, v)
    stride, blended = _tile_strides(case, v)
    H, W = v.height, v.width
    gw = stride.shape[1]
    # (tile, Gaussian) pairs, tile-major, Gaussians in index order
    nx, count = b[:, 1] - b[:, 0], (b[:, 1] - b[:, 0]) * (b[:, 3] - b[:, 2])
    prim = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    k = torch.arange(len(prim), device="cuda") - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
    tile = (b[prim, 2] + k // nx[prim]) * gw + b[prim, 0] + k % nx[prim]
    tile, order = torch.sort(tile, stable=True)
    prim = prim[order]
    length = torch.bincount(tile, minlength=stride.numel())
    begin = torch.cumsum(length, 0) - length
    work = torch.zeros(3, H, W, dtype=torch.float64, device="cuda")
    for s in (1, 2, 4):
        mine = (stride.reshape(-1) == s).nonzero().squeeze(1)
        if not len(mine):
            continue
        mine = mine[torch.argsort(length[mine], descending=True)]
        o = torch.arange(0, TILE, s, device="cuda")
        px = ((mine % gw) * TILE).unsqueeze(1) + o.repeat(len(o)).unsqueeze(0)
        py = ((mine // gw) * TILE).unsqueeze(1) + o.repeat_interleave(len(o)).unsqueeze(0)
        col = _blend(case, v, (P1, P2, P4, rgb, opacity), prim, begin[mine], length[mine], px, py, bg)
        ok = (px < W) & (py < H)
        work[:, py[ok], px[ok]] = col.permute(2, 0, 1)[:, ok]
    return _compose(case, v, work, stride, blended)


def _blend(case, v, rec, prim, begin, length, px, py, bg):
    """Colours [tiles, samples, 3] of the samples (px, py): one list position of all tiles a step."""
    P1, P2, P4, rgb, opacity = rec
    K, (n, m) = case["K"], px.shape
    x, y = px.double(), py.double()
    new = dict(dtype=torch.float64, device="cuda")
    depth = torch.full((n * m, K), 3.402823466e38, **new)
    core = torch.zeros(n * m, K, 4, **new)  # RGBA, quantised to 8 bits
    tail, T = torch.zeros(n, m, 4, **new), torch.ones(n, m, **new)
    lengths = length.cpu().numpy()
    active = np.searchsorted(-lengths, -np.arange(int(lengths[0]) if n else 0) - 0.5)  # tiles with length > t
    for t, a in enumerate(active.tolist()):
        p = prim[begin[:a] + t]
        A, B, C = P1[p].unsqueeze(1), P2[p].unsqueeze(1), P4[p].unsqueeze(1)
        plane_x, plane_y = A - C * x[:a, :, None], B - C * y[:a, :, None]
        nx, ny = plane_x[..., :3], plane_y[..., :3]
        mm = plane_x[..., 3:] * ny - nx * plane_y[..., 3:]
        d = torch.linalg.cross(nx, ny)
        num, den = (mm * mm).sum(-1), (d * d).sum(-1)
        alpha = (opacity[p].unsqueeze(1) * torch.exp(-0.5 * num / den)).clamp(max=1.0)
        frag = (num <= MAX_CUTOFF_SQ * den) & (alpha >= MIN_ALPHA)
        pm = torch.cat([rgb[p].unsqueeze(1) * alpha.unsqueeze(-1), alpha.unsqueeze(-1)], -1)
        z = (C[..., :3] * torch.linalg.cross(d, mm)).sum(-1) / den + C[..., 3]
        cand = frag & (alpha >= MIN_ALPHA_CORE) & (z < depth.view(n, m, K)[:a, :, K - 1])
        i = cand.reshape(-1).nonzero().squeeze(1)
        if len(i):
            fz, fc = z.reshape(-1)[i], torch.floor(pm.reshape(-1, 4)[i].clamp(0.0, 1.0) * 255.0 + 0.5) / 255.0
            dk, ck = depth[i], core[i]
            for q in range(K):
                first = fz < dk[:, q]
                z_q, c_q = dk[:, q].clone(), ck[:, q].clone()
                dk[:, q] = torch.where(first, fz, z_q)
                ck[:, q] = torch.where(first.unsqueeze(1), fc, c_q)
                fz, fc = torch.where(first, z_q, fz), torch.where(first.unsqueeze(1), c_q, fc)
            depth[i], core[i] = dk, ck
            pm.view(-1, 4)[i] = fc
        pm = torch.where(frag.unsqueeze(-1), pm, 0.0)
        tail[:a] += pm
        T[:a] *= 1.0 - pm[..., 3]
    out, Tc = torch.zeros(n, m, 3, **new), torch.ones(n, m, **new)
    core = core.view(n, m, K, 4)
    for q in range(K):
        on = Tc >= MIN_T
        out = torch.where(on.unsqueeze(-1), out + Tc.unsqueeze(-1) * core[:, :, q, :3], out)
        Tc = torch.where(on, Tc * (1.0 - core[:, :, q, 3]), Tc)
    some = (Tc >= MIN_T) & (tail[..., 3] >= MIN_ALPHA)
    weight = torch.where(some, Tc * (1.0 - T) / tail[..., 3].clamp(min=MIN_ALPHA), 0.0)
    out = out + weight.unsqueeze(-1) * tail[..., :3]
    if bg is not None:
        wb = Tc * T
        ray = torch.stack([x, y, torch.ones_like(x), torch.ones_like(x)], -1) @ _tensor(v.VPR_inv)[:3].T
        ray = ray / ray.norm(dim=-1, keepdim=True)
        colour = (torch.tanh(_sh_sum(bg, ray)) * 0.5 + 0.5).clamp(0.0, 1.0)
        fade = torch.where(ray[..., 1] > 0.1, 0.0, (1.0 - ray[..., 1] / 0.1).clamp(max=1.0))
        out = out + (torch.where(wb >= MIN_T, wb, 0.0) * fade).unsqueeze(-1) * colour
    return out.clamp(0.0, 1.0)


def _compose(case, v, work, stride, blended):
    """The image from the samples: strided tiles interpolated (or blurred), blended tiles faded."""
    H, W = work.shape[1:]
    y, x = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    ty, tx = y // TILE, x // TILE
    own = stride[ty, tx]
    fovea = (stride == 1) & ~blended
    src = work * (~fovea[ty, tx]) if case["blur"] else work
    out = torch.where(own == 1, work, 0.0)
    for s in (2, 4):
        mask = (own == s) | (blended[ty, tx] if s == 2 else False)
        if not bool(mask.any()):
            continue
        total = torch.zeros_like(work)
        fx, fy = (x % s).double() / s, (y % s).double() / s

        def weights(f):  # of the samples -1, 0, +1 from the pixel's own
            if not case["blur"]:
                return torch.zeros_like(f), 1.0 - f, f
            even = f == 0
            return torch.where(even, 0.125, 0.0), torch.where(even, 0.75, 0.5), torch.where(even, 0.125, 0.5)

        for dy, wy in zip((-1, 0, 1), weights(fy)):
            for dx, wx in zip((-1, 0, 1), weights(fx)):
                sx = ((x // s + dx) * s).clamp(0, (W - 1) // s * s)
                sy = ((y // s + dy) * s).clamp(0, (H - 1) // s * s)
                other = stride[sy // TILE, sx // TILE]
                foreign = (other == 0) | ((other == 4) if s == 2 else False)  # no such sample there
                cx = torch.minimum(torch.maximum(sx, tx * TILE), tx * TILE + TILE - s)
                cy = torch.minimum(torch.maximum(sy, ty * TILE), ty * TILE + TILE - s)
                sx, sy = torch.where(foreign, cx, sx), torch.where(foreign, cy, sy)
                total += src[:, sy, sx] * (wx * wy)
        total = total.clamp(0.0, 1.0)
        if s == 2:
            gaze = _tensor(v.gaze_position)
            far = torch.sqrt((gaze[0] - x) ** 2 + (gaze[1] - y) ** 2)
            fade = ((far - BLEND_TILES * TILE - TILE) / (BLEND_WIDTH_PX - TILE)).clamp(0.0, 1.0)
            faded = (total * fade + work * (1.0 - fade)).clamp(0.0, 1.0)
            total = torch.where(blended[ty, tx], faded, total)
        out = torch.where(mask, total, out)
    return out
