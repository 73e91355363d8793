"""The work a user has this framework do, as timed cases.

Every case goes through the public Python binding (``pilot_b200.beams``) the way
a visualisation program does: a renderer that is kept, a volume, a colour map,
lights and a camera, then a frame into the caller's image. The cases are the
forms a frame comes in (exact, lazily built map, 16-bit fields, bricks, a batch
of requests, the learned transmittance) and the network's own two directions.

Fields are seeded turbulence (octaves of trilinear value noise) or Gaussian
blobs, the two kinds of data of the benchmark; the colour map is its 256-entry
table. ``exact`` marches the same rays in float64 with plain torch.
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

from pilot_b200 import beams

IN, HID = 112, 64           # the transmittance network: 112 -> 4 x 64 (ReLU) -> 1 (sigmoid)
LIGHT_STEPS = 128           # light samples over the volume diagonal (the renderer's default)
DIAG = math.sqrt(3.0)       # every volume spans the unit cube


def _frame(name, kind, field, nx, ny, nz, width, height, cells, **more):
    case = {"name": name, "kind": kind, "field": field, "nx": nx, "ny": ny, "nz": nz, "width": width,
            "height": height, "cells": cells, "step": 0.5, "light": "point", "lights": 1, "cut": 0.99}
    case.update(more)
    return case


def listed():
    return [
        # the reference's own call: a host field through the mapper, image back on the host
        _frame("mapper_host", "mapper", "blobs", 96, 80, 112, 320, 240, 48),
        # an interactive preview: the smallest frame, bound by latency and launches
        _frame("preview", "frame", "blobs", 64, 64, 64, 256, 256, 32),
        # the ordinary scene of the tests and the benchmark: 128^3 blobs under a directional light
        _frame("blobs128", "frame", "blobs", 128, 128, 128, 512, 512, 128, light="directional"),
        # the headline frame: 512^3 turbulence, full 257^3-vertex map; turbulence has no empty
        # space, so this program has turned the empty-space skip off, as the autotuner does
        _frame("noise512", "frame", "noise", 512, 512, 512, 1024, 1024, 256, skip=False),
        # the same frame for a user who wants the image only
        _frame("lazy512", "lazy", "noise", 512, 512, 512, 1024, 1024, 256),
        # a running simulation: every frame brings a new field of ragged size, three lights
        _frame("timestep", "timestep", "blobnoise", 311, 257, 203, 801, 603, 96, lights=3),
        # a bfloat16 volume in the 16-bit form, finely sampled
        _frame("bf16_384", "precision", "blobnoise", 384, 384, 384, 1024, 1024, 192, step=0.25, dtype="bf16"),
        # a domain decomposed into blocks: local maps, stitching, per-block marches, composite
        _frame("bricks256", "bricks", "noise", 257, 257, 257, 768, 768, 64, splits=2),
        # serving: many requests of mixed sizes over resident volumes in one call
        {"name": "batch16", "kind": "batch", "requests": 16, "volumes": 4, "nmax": 192, "imax": 512},
        # the network's dense forward pass on a large set of feature rows
        {"name": "network_forward", "kind": "forward", "rows": 1000003},
        # a learned frame: the network shades, a probe check sends bad tiles to the exact map
        _frame("learned256", "learned", "noise", 256, 256, 256, 768, 768, 128),
        # training the network on a new volume
        _frame("training", "training", "noise", 160, 160, 160, 0, 0, 64, samples_log2=18, epochs=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Any form of frame at any size up to the listed ones, or a forward pass."""
    kind = rng.choice(["frame", "frame", "frame", "lazy", "timestep", "precision", "bricks", "mapper", "batch",
                       "forward"])
    if kind == "batch":
        return {"kind": kind, "requests": _log(rng, 2, 20), "volumes": rng.randint(1, 4),
                "nmax": rng.randint(64, 192), "imax": rng.randint(128, 512)}
    if kind == "forward":
        return {"kind": kind, "rows": _log(rng, 1000, 1500000)}
    top = {"mapper": 120, "bricks": 257}.get(kind, 400)
    n = [_log(rng, 24, top) for _ in range(3)]
    case = _frame("", kind, rng.choice(["noise", "blobs", "blobnoise"]), *n, _log(rng, 96, 1024), _log(rng, 96, 1024),
                  _log(rng, 12, 64 if kind == "bricks" else 192), step=rng.choice([0.25, 0.5, 0.7, 1.0]),
                  light=rng.choice(["point", "directional"]), cut=rng.choice([0.95, 0.99, 1.0]))
    del case["name"]
    if kind in ("frame", "timestep"):
        case["lights"] = rng.choice([1, 1, 1, 2, 3])
        case["skip"] = rng.random() < 0.7
        if case["lights"] == 1 and rng.random() < 0.2:
            case["rect"] = True
    if kind == "precision":
        case["dtype"] = rng.choice(["bf16", "f16"])
    if kind == "bricks":
        case["splits"] = 2
    return case


# -- inputs ----------------------------------------------------------------------

def _field(case, seed, kind=None, dims=None):
    """The scalar field, float32 (z, y, x) on the GPU, normalised to [0, 1]."""
    nx, ny, nz = dims or (case["nx"], case["ny"], case["nz"])
    kind = kind or case["field"]
    g = torch.Generator().manual_seed(seed * 7919 + 13)

    def noise():
        v = torch.zeros((1, 1, nz, ny, nx), device="cuda")
        for o in range(4):
            k = (6 << o) + 1
            grid = torch.rand((1, 1, k, k, k), generator=g).mul_(2).sub_(1).mul_(0.5 ** o).cuda()
            v += F.interpolate(grid, size=(nz, ny, nx), mode="trilinear", align_corners=True)
        return v[0, 0]

    def blobs(count):
        p = torch.rand((count, 5), generator=g).double()
        ax = [torch.linspace(0, 1, m, dtype=torch.float64) for m in (nz, ny, nx)]
        s = 0.05 + 0.1 * p[:, 3:4]
        e = [torch.exp(-(a[None, :] - (0.2 + 0.6 * p[:, 2 - d:3 - d])) ** 2 / (2 * s * s)) for d, a in enumerate(ax)]
        e[0] = e[0] * (0.5 + 0.5 * p[:, 4:5])
        e = [a.float().cuda() for a in e]
        v = torch.zeros((nz, ny, nx), device="cuda")
        for b in range(count):
            v += e[0][b][:, None, None] * e[1][b][None, :, None] * e[2][b][None, None, :]
        return v

    if kind == "noise":
        v = noise()
    elif kind == "blobs":
        v = blobs(8)
    else:
        v = blobs(24)
        v /= v.max()
        v += 0.1 * noise()
    lo, hi = v.min(), v.max()
    return ((v - lo) * (1.0 / (hi - lo))).clamp_(0, 1).contiguous()


def _colour_map():
    v = np.arange(256) / 255.0
    alpha = np.interp(v, (0.2, 0.4, 0.6, 0.8), (0.0, 0.05, 0.2, 0.6))
    rgb = np.array([0.23, 0.30, 0.75])[None] * (1 - v)[:, None] + np.array([0.95, 0.55, 0.10])[None] * v[:, None]
    return np.concatenate([rgb, alpha[:, None]], axis=1).astype(np.float32)


def _unit(rng):
    while True:
        v = [rng.gauss(0, 1) for _ in range(3)]
        n = math.sqrt(sum(x * x for x in v))
        if n > 1e-3:
            return [x / n for x in v]


def _view(case, seed):
    """Camera, lights and, for a rectilinear grid, the axes' coordinates."""
    rng = random.Random(seed * 104729 + 7)
    d = _unit(rng)
    view = {"eye": [0.5 + x for x in d], "up": [0.0, 1.0, 0.0] if abs(d[1]) < 0.9 else [1.0, 0.0, 0.0],
            "fov": 30.0, "lights": []}
    for k in range(case.get("lights", 1)):
        u = _unit(rng)
        at = u if case["light"] == "directional" else [0.5 + 2.0 * DIAG * x for x in u]
        view["lights"].append((at, [1.0, 0.9 - 0.2 * k, 0.6 + 0.2 * k]))
    if case.get("rect"):
        view["axes"] = []
        for m in (case["nx"], case["ny"], case["nz"]):
            w = [rng.uniform(0.6, 1.4) for _ in range(m - 1)]
            c = np.concatenate([[0.0], np.cumsum(w)]) / sum(w)
            view["axes"].append(c.astype(np.float32))
    return view


def _distance(case):
    return case["step"] / (max(case["nx"], case["ny"], case["nz"]) - 1)


def _spacing(case):
    return tuple(1.0 / (m - 1) for m in (case["nx"], case["ny"], case["nz"]))


def _camera(case, view):
    return beams.Renderer.camera(view["eye"], (0.5, 0.5, 0.5), view["up"], view["fov"], case["width"], case["height"])


def _renderer(case, view):
    r = beams.Renderer(0)
    r.set_color_map(_colour_map())
    r.set_shadow_map_size(case["cells"])
    r.set_sample_distance(_distance(case))
    r.set_termination_alpha(case["cut"])
    for at, colour in view["lights"]:
        if case["light"] == "point":
            r.add_point_light(at, colour)
        else:
            r.add_directional_light(at, colour)
    if len(view["lights"]) > 1:
        r.set_multi_light(True)
    if not case.get("skip", True):
        r.set_tuning(light_brick=8, empty_skip=False, view_skip=False)
    return r


def _batch(case, seed):
    """The batch's requests as frames of their own: (volume, frame case, view)."""
    rng = random.Random(seed * 31337 + 3)
    sizes = [max(24, int(case["nmax"] * f)) for f in (1.0, 0.66, 0.5, 0.33)][:case["volumes"]]
    kinds = ["blobs" if i % 2 else "noise" for i in range(case["volumes"])]
    reqs = []
    for i in range(case["requests"]):
        v = i % case["volumes"]
        n = sizes[v]
        im = max(64, case["imax"] // (1 + i % 3))
        fc = _frame("", "frame", kinds[v], n, n, n, im, im - 7 * (i % 2), n // 2)
        reqs.append((v, fc, _view(fc, rng.randrange(1 << 30))))
    return sizes, kinds, reqs


def _network(seed):
    """Parameters of a network of the trained one's shape and scale, one flat float32 vector."""
    g = torch.Generator().manual_seed(seed + 5)
    parts = []
    for i, fan in enumerate((IN, HID, HID, HID)):
        parts += [(torch.rand(fan * HID, generator=g) * 2 - 1) * math.sqrt(6.0 / fan),
                  (torch.rand(HID, generator=g) - 0.5) * 0.2]
    parts += [(torch.rand(HID, generator=g) * 2 - 1) * 0.2, torch.tensor([1.0])]
    return torch.cat(parts)


def _features(case, seed):
    """Encoded samples: positions and light directions in [-1, 1], then sines and cosines, 10 columns unused."""
    g = torch.Generator(device="cuda").manual_seed(seed + 11)
    x = torch.rand((case["rows"], IN), generator=g, device="cuda") * 2 - 1
    x[:, 102:] = 0
    return x.bfloat16()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "forward":
        s["r"] = beams.Renderer(0)
        s["r"].mlp_set_params(_network(seed).numpy())
        s["x"] = _features(case, seed)
        s["T"] = torch.empty(case["rows"], device="cuda")
        return s
    if kind == "batch":
        sizes, kinds, reqs = _batch(case, seed)
        r = s["r"] = beams.Renderer(0)
        r.set_color_map(_colour_map())
        s["fields"] = [_field(None, seed + i, k, (n, n, n)) for i, (n, k) in enumerate(zip(sizes, kinds))]
        r.batch_set_volumes([(f, (0, 0, 0), (1.0 / (n - 1),) * 3, (0, 1)) for f, n in zip(s["fields"], sizes)])
        s["reqs"] = [r.request(v, _camera(fc, view), view["lights"][0][0], 0, view["lights"][0][1], 1.0, fc["cells"],
                               _distance(fc), fc["cut"],
                               out=torch.empty((fc["height"], fc["width"], 4), device="cuda"))
                     for v, fc, view in reqs]
        return s
    view = _view(case, seed)
    field = s["field"] = _field(case, seed)
    if kind == "mapper":
        m = s["m"] = beams.MapperLightedVolume(0)
        m.SetCanvas(case["width"], case["height"])
        m.SetShadowMapSize(case["cells"])
        m.SetSampleDistance(_distance(case))
        m.SetActiveColorTable(_colour_map())
        m.renderer.set_termination_alpha(case["cut"])
        at, colour = view["lights"][0]
        if case["light"] == "point":
            m.AddLight(at, colour)
        else:
            m.renderer.add_directional_light(at, colour)
        s["field"] = field.cpu().numpy()
        s["spacing"] = _spacing(case)
        s["camera"] = {"position": view["eye"], "look_at": (0.5, 0.5, 0.5), "up": view["up"], "fov_y_deg": view["fov"]}
        return s
    r = s["r"] = _renderer(case, view)
    if kind == "training":
        r.set_volume(field)
        s["opts"] = beams.mlp_options(samples_log2=case["samples_log2"], n_lights=8, epochs=case["epochs"], batch=8192,
                                      seed=seed % 1000 + 1)
        return s
    s["cam"] = _camera(case, view)
    s["out"] = torch.empty((case["height"], case["width"], 4), device="cuda")
    if kind == "bricks":
        h = _spacing(case)
        cut = [[round(i * (m - 1) / case["splits"]) for i in range(case["splits"] + 1)]
               for m in (case["nx"], case["ny"], case["nz"])]
        s["bricks"] = []
        for z0, z1 in zip(cut[2], cut[2][1:]):
            for y0, y1 in zip(cut[1], cut[1][1:]):
                for x0, x1 in zip(cut[0], cut[0][1:]):
                    sub = field[z0:z1 + 1, y0:y1 + 1, x0:x1 + 1].contiguous()
                    s["bricks"].append((sub, (x0 * h[0], y0 * h[1], z0 * h[2]), h, (0, 1)))
        r.set_bricks(s["bricks"])
        return s
    if kind == "precision":
        s["field"] = field = field.to(torch.bfloat16 if case["dtype"] == "bf16" else torch.float16)
        r.set_form(beams.FORM_PRECISION, beams.BF16 if case["dtype"] == "bf16" else beams.F16)
    r.set_volume(field)
    if "axes" in view:
        s["axes"] = view["axes"]
        r.set_volume_coordinates(*view["axes"])
    if kind == "lazy":
        r.set_lazy_shadow_map(True)
    if kind == "learned":
        r.mlp_train(beams.mlp_options(samples_log2=18, n_lights=2, epochs=2, batch=4096, scene_light=1, seed=3))
        r.set_form(beams.FORM_MLP, beams.mlp_options(knot=8, fallback_tol=0.05))
    return s


def run(s):
    kind = s["kind"]
    if kind == "forward":
        s["r"].mlp_forward_tc_device(s["x"], s["T"])
        return s["T"]
    if kind == "batch":
        return s["r"].render_batch(s["reqs"], timings=False)[0]
    if kind == "mapper":
        return s["m"].RenderCells(s["field"], (0, 0, 0), s["spacing"], (0, 1), s["camera"])
    if kind == "training":
        report = s["r"].mlp_train(s["opts"])
        return {"params": s["r"].mlp_params(), "holdout_rmse": report["holdout_rmse"]}
    if kind == "timestep":  # this step's field
        s["r"].set_volume(s["field"])
        if "axes" in s:
            s["r"].set_volume_coordinates(*s["axes"])
    return s["r"].render(s["cam"], s["out"], timings=False)[0]


def _frame_work(case):
    """A light ray meets on average half a volume crossing (about 0.9 of an edge) before its vertex, a
    view ray up to a whole one over the part of the image the volume covers; some 45 operations a light
    sample (trilinear value, table index, accumulate) and 70 a view sample (two trilinear values, shading)."""
    cells = case["cells"]
    vertices = (cells + 1) ** 3 * case.get("lights", 1) * (0.05 if case["kind"] == "lazy" else 1.0)
    light = vertices * 0.45 / DIAG * LIGHT_STEPS
    view = 0.3 * case["width"] * case["height"] * 0.9 / _distance(case)
    size = 2 if case["kind"] == "precision" else 4
    return (case["nx"] * case["ny"] * case["nz"] * size + case["width"] * case["height"] * 16,
            45 * light + 70 * view)


def work(case):
    kind = case["kind"]
    if kind == "forward":
        macs = IN * HID + 3 * HID * HID + HID
        return {"bytes": case["rows"] * (2 * IN + 4), "flops": 2 * macs * case["rows"]}
    if kind == "training":
        rows = 1 << case["samples_log2"]
        macs = IN * HID + 3 * HID * HID + HID
        light = rows * 0.45 / DIAG * LIGHT_STEPS
        return {"bytes": case["nx"] * case["ny"] * case["nz"] * 4 + 4 * macs,
                "flops": 45 * light + 6 * macs * rows * case["epochs"]}
    if kind == "batch":
        sizes, _, reqs = _batch(case, 0)
        parts = [_frame_work(fc) for _, fc, _ in reqs]
        images = sum(fc["width"] * fc["height"] * 16 for _, fc, _ in reqs)
        return {"bytes": sum(4 * n ** 3 for n in sizes) + images, "flops": sum(f for _, f in parts)}
    b, f = _frame_work(case)
    return {"bytes": b, "flops": f}


# -- the same outputs in 64 bits ----------------------------------------------------

def _trilinear(field, cell, frac):
    """field (z, y, x) float64; cell and frac: three tensors each, x y z."""
    nz, ny, nx = field.shape
    flat = field.reshape(-1)
    base = (cell[2] * ny + cell[1]) * nx + cell[0]
    x, y, z = frac

    def row(off):
        a = flat[base + off]
        return a + x * (flat[base + off + 1] - a)

    def face(off):
        a = row(off)
        return a + y * (row(off + nx) - a)

    a = face(0)
    return a + z * (face(nx * ny) - a)


def _locate(p, axes, n):
    """Cell and fraction of positions p (three tensors in [0, 1]) on uniform or explicit axes."""
    cell, frac = [], []
    for d in range(3):
        if axes is None:
            t = p[d] * (n[d] - 1)
            c = t.long().clamp_(0, n[d] - 2)
            cell.append(c)
            frac.append(t - c)
        else:
            c = (torch.searchsorted(axes[d], p[d].contiguous(), right=True) - 1).clamp_(0, n[d] - 2)
            lo = axes[d][c]
            cell.append(c)
            frac.append((p[d] - lo) / (axes[d][c + 1] - lo))
    return cell, frac


def _inside(p):
    ok = (p[0] >= 0) & (p[0] <= 1)
    for d in (1, 2):
        ok &= (p[d] >= 0) & (p[d] <= 1)
    return ok


def _slab(origin, direction):
    """Entry and exit distances of the unit cube."""
    lo, hi = None, None
    for d in range(3):
        a, b = (0.0 - origin[d]) / direction[d], (1.0 - origin[d]) / direction[d]
        n, f = torch.minimum(a, b), torch.maximum(a, b)
        lo = n if lo is None else torch.maximum(lo, n)
        hi = f if hi is None else torch.minimum(hi, f)
    return lo, hi


def _opacity_map(field, axes, alpha, cells, light, directional):
    """Opacity of the light's march to every vertex of the (cells + 1)^3 grid."""
    n = (field.shape[2], field.shape[1], field.shape[0])
    m = cells + 1
    step = DIAG / LIGHT_STEPS
    out = torch.empty(m ** 3, dtype=torch.float64, device="cuda")
    chunk = 1 << 22
    for first in range(0, m ** 3, chunk):
        ids = torch.arange(first, min(first + chunk, m ** 3), device="cuda")
        V = [(ids % m).double() / cells, (ids // m % m).double() / cells, (ids // (m * m)).double() / cells]
        L = [V[d] - 2 * DIAG * light[d] for d in range(3)] if directional else \
            [torch.full_like(V[0], light[d]) for d in range(3)]
        length = torch.sqrt(sum((V[d] - L[d]) ** 2 for d in range(3)))
        u = [(V[d] - L[d]) / length for d in range(3)]
        t0, t1 = _slab(L, u)
        t0, t1 = t0.clamp(min=0), torch.minimum(t1, length)
        o = torch.zeros_like(length)
        live = torch.ones_like(length, dtype=torch.bool)
        for k in range(LIGHT_STEPS + 8):
            live = live & ((k * step) ** 2 <= (t1 - t0) ** 2)  # a vertex on the entry face takes one sample
            t = t0 + (k + 1) * step
            p = [L[d] + t * u[d] for d in range(3)]
            live = live & _inside(p)
            if k % 16 == 0 and not bool(live.any()):
                break
            c, f = _locate([q.clamp(0, 1) for q in p], axes, n)
            i = (_trilinear(field, c, f) * 255).long().clamp_(0, 255)
            o = torch.where(live, o + (1 - o) * alpha[i], o)
        out[first:first + chunk] = o
    return out.reshape(m, m, m)


def _exact_frame(case, view, field):
    field = field.double()
    tf = torch.from_numpy(_colour_map()).double().cuda()
    axes = [torch.from_numpy(a).double().cuda() for a in view["axes"]] if "axes" in view else None
    n = (case["nx"], case["ny"], case["nz"])
    cells, sd = case["cells"], _distance(case)
    directional = case["light"] == "directional"
    maps = []
    for at, colour in view["lights"]:
        size = math.sqrt(sum(x * x for x in at))
        at = [x / size for x in at] if directional else at
        maps.append((_opacity_map(field, axes, tf[:, 3] / tf[:, 3].max(), cells, at, directional), colour))
    w, h = case["width"], case["height"]
    eye = torch.tensor(view["eye"], dtype=torch.float64)
    fwd = F.normalize(torch.tensor([0.5] * 3, dtype=torch.float64) - eye, dim=0)
    right = F.normalize(torch.linalg.cross(fwd, torch.tensor(view["up"], dtype=torch.float64)), dim=0)
    up = torch.linalg.cross(right, fwd)
    th = math.tan(math.radians(view["fov"] / 2))
    y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    sx = ((x.reshape(-1).double() + 0.5) * (2 / w) - 1) * th * w / h
    sy = ((y.reshape(-1).double() + 0.5) * (2 / h) - 1) * th
    v = [fwd[d].item() + sx * right[d].item() + sy * up[d].item() for d in range(3)]
    size = torch.sqrt(sum(a * a for a in v))
    u = [a / size for a in v]
    o = [torch.full_like(sx, eye[d].item()) for d in range(3)]
    t0, t1 = _slab(o, u)
    t0 = t0.clamp(min=0)
    image = torch.zeros((w * h, 4), dtype=torch.float64, device="cuda")
    ray = torch.nonzero(t1 >= t0).reshape(-1)
    o, u = [a[ray] for a in o], [a[ray] for a in u]
    t0, t1 = t0[ray], t1[ray]
    colour = torch.zeros((ray.numel(), 4), dtype=torch.float64, device="cuda")
    entered = torch.zeros_like(t0, dtype=torch.bool)
    k = 0
    while ray.numel():
        t = t0 + DIAG * 1e-4 + k * sd
        p = [o[d] + t * u[d] for d in range(3)]
        inside = _inside(p)
        entered |= inside
        live = inside & (t < t1) & (colour[:, 3] < case["cut"])
        if k % 32 == 0:  # keep the rays that still march
            on = live | (~entered & (t < t1))
            image[ray[~on]] = colour[~on]
            ray, t0, t1, colour, entered = ray[on], t0[on], t1[on], colour[on], entered[on]
            o, u, p, live = [a[on] for a in o], [a[on] for a in u], [a[on] for a in p], live[on]
        q = [a.clamp(0, 1) for a in p]
        c, f = _locate(q, axes, n)
        e = tf[(_trilinear(field, c, f) * 255).long().clamp_(0, 255)]
        a = torch.where(live, e[:, 3] * (1 - colour[:, 3]), torch.zeros_like(t0))
        c, f = _locate(q, None, (cells + 1,) * 3)
        shade = torch.zeros((ray.numel(), 3), dtype=torch.float64, device="cuda")
        for m, tint in maps:
            shade += (1 - _trilinear(m, c, f))[:, None] * torch.tensor(tint, dtype=torch.float64, device="cuda")
        colour[:, :3] += (e[:, :3] * shade).clamp_(0, 1) * a[:, None]
        colour[:, 3] += a
        k += 1
    return image.reshape(h, w, 4)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bricks", "learned"):  # their images depend on the decomposition and on trained weights
        return None
    if kind == "training":
        return None
    if kind == "forward":
        p = _network(seed).double().cuda()
        h = _features(case, seed).double()
        at = 0
        for fan in (IN, HID, HID, HID):
            w, b = p[at:at + fan * HID].reshape(fan, HID), p[at + fan * HID:at + fan * HID + HID]
            at += fan * HID + HID
            h = torch.relu(h @ w + b)
        return torch.sigmoid(h @ p[at:at + HID] + p[at + HID])
    if kind == "batch":
        sizes, kinds, reqs = _batch(case, seed)
        fields = [_field(None, seed + i, k, (n, n, n)) for i, (n, k) in enumerate(zip(sizes, kinds))]
        return [_exact_frame(fc, view, fields[v]) for v, fc, view in reqs]
    field = _field(case, seed)
    if kind == "precision":
        field = field.to(torch.bfloat16 if case["dtype"] == "bf16" else torch.float16)
    image = _exact_frame(case, _view(case, seed), field)
    return image.cpu().numpy() if kind == "mapper" else image
