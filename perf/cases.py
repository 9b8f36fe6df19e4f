"""Performance cases of the path-tracing core, through its Python entry points.

Each case is a dict of plain values. ``listed()`` names the workloads that are
followed over time, ``draw(rng)`` gives more of the same ranges, ``prepare``
makes what a caller has in hand before the call (device inputs, the scene, the
network), ``run`` is one pass, ``work`` its unavoidable bytes and operations,
and ``exact`` what the pass returns, in 64-bit arithmetic, where plain torch can
say.

The kinds of a case:

* ``trace``: closest-hit or any-hit queries over a soup of icospheres (picking,
  probes, visibility, the ray-cast benchmark).
* ``frame``: one dr_render call, the box room or the many-light scene: the
  interactive frame (one sample per pixel) and the offline image (many).
* ``batch``: images of several scenes of uneven size in one schedule.
* ``guided``: dr_render_guided with a network that has finished training.
* ``infer`` / ``train``: the guiding network by itself.
* ``alias``: the device build of a light table.
* ``tonemap``: the display conversion of an accumulated image.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from devilray_gb300 import native, scenes

LAYERS = ((80, 64), (64, 64), (64, 64), (64, 64), (64, 48))  # fan-in, fan-out of the guiding network


def listed() -> list:
    return [
        # the ray-cast benchmark: 2^20 triangles, 16.8 M incoherent rays
        _trace("trace_closest_16m", "closest", "reference", 1 << 20, 1 << 24),
        # a handful of picking / probe rays against a small model: launch latency
        _trace("trace_closest_pick", "closest", "reference", 5120, 1021),
        # visibility of a large set of segments, watertight test, no round count
        _trace("trace_any_4m", "any", "watertight", 300000, 4000037),
        # an interactive frame as the reference renders it: 256 x 256, one
        # sample per pixel and call, paths of up to 10 vertices
        _frame("frame_box_256", "box", 0, 256, 256, 1, 10),
        # the box-room image of the plain-method configuration: 16 spp, depth 8
        _frame("frame_box_256_16spp", "box", 0, 256, 256, 16, 8),
        # the many-light scene at 1080p (2^20 triangles, 65,536 emitters)
        _frame("frame_lights_1080p", "lights", 1 << 20, 1920, 1080, 4, 16),
        # images of eight uneven scenes in one schedule
        {"name": "batch_8_uneven", "kind": "batch", "scenes": 8, "tris_max": 200000, "res_max": 512, "spp": 4,
         "depth": 12},
        # a guided render with a finished network, the first three bounces guided
        {"name": "guided_480x270", "kind": "guided", "tris": 1 << 18, "width": 480, "height": 270, "spp": 16,
         "depth": 16, "bounces": 3},
        # the guiding network: the vertices of one bounce of a large wave
        {"name": "infer_1m", "kind": "infer", "rows": 1 << 20},
        # training from given parameters: the 16 Adam steps of 65,536 samples that
        # follow one wave of a guided render
        {"name": "train_16x64k", "kind": "train", "rows": 65536, "steps": 16},
        # the light table of a many-light scene
        {"name": "alias_66k", "kind": "alias", "weights": 66356},
        # the display image of a 1080p accumulation buffer
        {"name": "tonemap_1080p", "kind": "tonemap", "width": 1920, "height": 1080},
    ]


def _trace(name, query, test, tris, rays):
    return {"name": name, "kind": "trace", "query": query, "test": test, "tris": tris, "rays": rays}


def _frame(name, scene, tris, width, height, spp, depth):
    return {"name": name, "kind": "frame", "scene": scene, "tris": tris, "width": width, "height": height, "spp": spp,
            "depth": depth}


def draw(rng) -> dict:
    """One more case; sizes are uniform in their logarithm."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trace", "trace", "trace", "frame", "frame", "frame", "batch", "guided", "infer", "train",
                       "alias", "tonemap"])
    if kind == "trace":
        return {"kind": kind, "query": rng.choice(["closest", "any"]), "test": rng.choice(["reference", "watertight"]),
                "tris": size(256, 1 << 20), "rays": size(200, 1 << 24)}
    if kind == "frame":
        w = size(64, 1920)
        h = max(33, int(w * rng.uniform(0.5, 1.0)))
        spp = max(1, min(size(1, 16), (8 << 20) // (w * h)))
        scene = rng.choice(["box", "lights"])
        return {"kind": kind, "scene": scene, "tris": size(4096, 1 << 20) if scene == "lights" else 0, "width": w,
                "height": h, "spp": spp, "depth": rng.randint(2, 16)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 8), "tris_max": size(4000, 200000), "res_max": size(128, 512),
                "spp": rng.randint(1, 4), "depth": rng.randint(2, 12)}
    if kind == "guided":
        w = size(96, 480)
        return {"kind": kind, "tris": size(16384, 1 << 18), "width": w, "height": max(33, int(w * rng.uniform(0.5, 0.6))),
                "spp": rng.randint(1, 16), "depth": rng.randint(3, 16), "bounces": rng.randint(1, 4)}
    if kind == "infer":
        return {"kind": kind, "rows": size(1, 1 << 20)}
    if kind == "train":
        return {"kind": kind, "rows": size(512, 65536), "steps": rng.randint(1, 16)}
    if kind == "alias":
        return {"kind": kind, "weights": size(3, 1 << 20)}
    return {"kind": kind, "width": size(100, 3840), "height": size(60, 2160)}


# ---- inputs ---------------------------------------------------------------------------


def _gen(seed: int, stream: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + stream)


def _rand(g, *shape) -> torch.Tensor:
    return torch.rand(shape, generator=g, device="cuda")


def _unit(g, n: int) -> torch.Tensor:
    return torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)


def _soup(case, seed):
    half = scenes.density_half(case["tris"])
    soup, centres, radii = scenes.incoherent_soup(case["tris"], seed=seed, half=half)
    return soup, centres, radii, half


def _rays(case, seed, half) -> torch.Tensor:
    """dr_ray records: origins in the cube, directions on the sphere; any-hit
    rays are segments of up to the cube's width."""
    n = case["rays"]
    g = _gen(seed, 1)
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 0:3] = (2.0 * _rand(g, n, 3) - 1.0) * half
    rays[:, 4:7] = _unit(g, n)
    rays[:, 3] = _rand(g, n) * (2.0 * half) if case["query"] == "any" else math.inf
    return rays


def _materials(n: int) -> np.ndarray:
    return np.zeros((n, 16), np.float32)  # kind, ior, -, -, emission, albedo, debug colour: 4 floats each


def _lit_soup(tris: int, emitters: int, seed: int, half: float, above: float | None = None):
    """The many-light scene as arrays (positions, objects, materials): a seeded
    choice of triangles emits (each an object of its own), the other triangles
    of a sphere are one object, diffuse or glass. With `above`, only spheres
    whose centre lies above that height emit."""
    soup, centres, _ = scenes.incoherent_soup(tris, seed=seed, half=half)
    rng = np.random.default_rng(seed + 17)
    sphere = np.arange(tris) // 1280
    nsph = int(sphere[-1]) + 1
    can = np.arange(tris) if above is None else np.flatnonzero(centres[sphere, 1] > above)
    if can.size == 0:
        can = np.arange(tris)
    emissive = np.zeros(tris, bool)
    emissive[rng.permutation(can)[:emitters]] = True
    order = np.lexsort((np.arange(tris), emissive, sphere))  # a sphere's body, then its emitters
    soup, sphere, emissive = soup[order], sphere[order], emissive[order]
    begin = np.flatnonzero(np.concatenate([[True], (sphere[1:] != sphere[:-1]) | emissive[1:] | (emissive[1:] != emissive[:-1])]))
    count = np.diff(np.append(begin, tris))
    mats = _materials(len(begin))
    lit = emissive[begin]
    glass = (rng.random(nsph) < 0.5)[sphere[begin]] & ~lit
    mats[:, 0] = np.where(glass, 1, 0).astype(np.int32).view(np.float32)
    mats[:, 1] = np.where(glass, rng.uniform(1.3, 1.7, nsph)[sphere[begin]], 0.0)
    mats[:, 4:7] = np.where(lit, np.exp(rng.normal(0.0, 1.5, len(begin))), 0.0)[:, None]
    mats[:, 8:11] = np.where(lit | glass, 0.0, rng.uniform(0.2, 0.8, nsph)[sphere[begin]])[:, None]
    objs = np.zeros(len(begin), [("tri_begin", "<u4"), ("tri_count", "<u4"), ("material", "<i4"), ("surface_area", "<f4")])
    objs["tri_begin"], objs["tri_count"], objs["material"] = begin, count, np.arange(len(begin))
    objs["surface_area"] = np.add.reduceat(scenes.tri_area_f32(soup).astype(np.float64), begin)
    return soup, objs, mats


def _add_room(soup, objs, mats, half: float):
    """The slab, floor, walls and ceiling of the guided configuration."""
    w = 1.15 * half
    parts = [scenes.rect_y(-w + 0.15 * half, w, -w, w, 0.3 * half)]
    for c, n, r in (((0, -w, 0), (0, 1, 0), (1, 0, 0)), ((0, 0, w), (0, 0, -1), (1, 0, 0)),
                    ((-w, 0, 0), (1, 0, 0), (0, 0, 1)), ((w, 0, 0), (-1, 0, 0), (0, 0, 1)),
                    ((0, w, 0), (0, -1, 0), (1, 0, 0))):
        parts.append(scenes.quad(c, n, r, 2 * w))
    grey = _materials(1)
    grey[:, 8:11] = 0.4
    more = np.zeros(len(parts), objs.dtype)
    more["tri_begin"] = soup.shape[0] + 2 * np.arange(len(parts))
    more["tri_count"] = 2
    more["material"] = len(mats)
    more["surface_area"] = [scenes.surface_area(p) for p in parts]
    return np.concatenate([soup, *parts]), np.concatenate([objs, more]), np.concatenate([mats, grey])


def _net(seed: int) -> np.ndarray:
    """Parameters of a guiding network: He-uniform layers, output biases that
    spread the lobes' concentrations and directions."""
    rng = np.random.default_rng(seed + 99)
    parts = []
    for i, (fan_in, fan_out) in enumerate(LAYERS):
        bound = math.sqrt(6.0 / fan_in) * (0.1 if i == 4 else 1.0)
        parts.append(rng.uniform(-bound, bound, fan_in * fan_out))
        parts.append(rng.normal(0.0, 1.0, fan_out) if i == 4 else np.zeros(fan_out))
    return np.concatenate(parts).astype(np.float32)


def _samples(case, seed):
    """Rows of the guiding network: positions, normals, and the directions and
    weights of the training samples, `steps` batches."""
    n = case["rows"] * case.get("steps", 1)
    g = _gen(seed, 2)
    pos = (2.0 * _rand(g, n, 3) - 1.0) * 50.0
    nrm, sdir = _unit(g, n), _unit(g, n)
    weight = torch.exp(torch.randn(n, generator=g, device="cuda"))
    return pos, nrm, sdir, weight


def _batch_sizes(case):
    """Triangles and image width of each scene: spread over the logarithm, the
    largest scene with the smallest image."""
    n = case["scenes"]
    tris = np.geomspace(1000.0, case["tris_max"], n).astype(int)
    res = np.geomspace(case["res_max"], 64.0, n).astype(int)
    return tris, res


def _image(width: int, height: int):
    n = width * height
    return torch.zeros((n, 4), device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    ctx = native.Context(0)
    if kind == "trace":
        soup, _, _, half = _soup(case, seed)
        n = case["rays"]
        out = torch.empty((n, 2), dtype=torch.int32, device="cuda") if case["query"] == "closest" else \
            torch.empty(n, dtype=torch.uint8, device="cuda")
        mode = native.DR_TRI_WATERTIGHT if case["test"] == "watertight" else native.DR_TRI_REFERENCE
        return {"case": case, "ctx": ctx, "scene": native.Scene(ctx, soup), "rays": _rays(case, seed, half), "out": out,
                "mode": mode}
    if kind == "frame":
        w, h = case["width"], case["height"]
        if case["scene"] == "box":
            m = np.eye(4, dtype=np.float32)
            m[0, 3] = 0.02 * np.random.default_rng(seed).uniform(-1, 1)
            scene = native.Scene.from_spec(ctx, scenes.box_room(3))
            cam = scenes.camera(w, h, transform=m)
        else:
            half = scenes.density_half(case["tris"])
            soup, objs, mats = _lit_soup(case["tris"], max(16, case["tris"] // 16), seed, half)
            scene = native.Scene(ctx, soup, objects=objs, materials=mats)
            cam = scenes.outside_camera(w, h, distance=3.0 * half, half=half)
        accum, casts = _image(w, h)
        return {"case": case, "ctx": ctx, "scene": scene, "cam": cam, "accum": accum, "casts": casts, "seed": seed}
    if kind == "batch":
        n = case["scenes"]
        tris, res = _batch_sizes(case)
        keep, jobs, images = [], [], []
        for i in range(n):
            half = scenes.density_half(int(tris[i]))
            soup, objs, mats = _lit_soup(int(tris[i]), max(16, int(tris[i]) // 64), seed + i, half)
            scene = native.Scene(ctx, soup, objects=objs, materials=mats)
            r = int(res[i])
            accum, casts = _image(r, r)
            cam = scenes.outside_camera(r, r, distance=3.0 * half, half=half)
            jobs.append(native.make_job(scene, cam, accum, casts, spp=case["spp"], max_depth=case["depth"], seed=seed))
            keep.append(scene)
            images.append((accum, casts))
        return {"case": case, "ctx": ctx, "scenes": keep, "batch": native.Batch(ctx, jobs), "images": images}
    if kind == "guided":
        half = scenes.density_half(case["tris"])
        arrays = _lit_soup(case["tris"], case["tris"] // 16, seed, half, above=0.4 * half)
        soup, objs, mats = _add_room(*arrays, half)
        guide = native.Guide(ctx, seed=seed, half_extent=1.2 * half)
        guide.set_params(_net(seed))
        w, h = case["width"], case["height"]
        accum, casts = _image(w, h)
        return {"case": case, "ctx": ctx, "scene": native.Scene(ctx, soup, objects=objs, materials=mats),
                "guide": guide, "cam": scenes.lower_camera(w, h, distance=3.0 * half, half=half), "accum": accum,
                "casts": casts, "seed": seed}
    if kind in ("infer", "train"):
        guide = native.Guide(ctx, seed=seed, half_extent=50.0)
        net = _net(seed)
        guide.set_params(net)
        pos, nrm, sdir, weight = _samples(case, seed)
        state = {"case": case, "ctx": ctx, "guide": guide, "net": net, "pos": pos, "nrm": nrm}
        if kind == "infer":
            state["y"] = torch.empty((case["rows"], 40), device="cuda")
        else:
            state.update(sdir=sdir, weight=weight)
        return state
    if kind == "alias":
        n = case["weights"]
        g = _gen(seed, 3)
        weights = torch.exp(1.5 * torch.randn(n, generator=g, device="cuda"))
        weights[_rand(g, n) < 0.02] = 0.0  # objects that do not emit
        return {"case": case, "ctx": ctx, "weights": weights,
                "table": torch.empty((n, 5), dtype=torch.int32, device="cuda")}
    n = case["width"] * case["height"]
    g = _gen(seed, 4)
    accum = torch.empty((n, 4), device="cuda")
    spp = 64.0
    accum[:, :3] = spp * torch.exp(1.2 * torch.randn((n, 3), generator=g, device="cuda") - 1.5)
    accum[_rand(g, n) < 0.03] = 0.0  # pixels whose paths met no light, or beyond the scene
    accum[:, 3] = spp
    return {"case": case, "ctx": ctx, "accum": accum, "rgba": torch.empty(n, dtype=torch.int32, device="cuda")}


# ---- one pass -------------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "trace":
        out = state["out"]
        if case["query"] == "any":
            state["scene"].trace_any(state["rays"], case["rays"], out, state["mode"])
            return {"occluded": out}
        state["scene"].trace_closest(state["rays"], case["rays"], out, state["mode"])
        return {"t": out[:, 0].view(torch.float32), "prim": out[:, 1]}
    if kind == "frame":
        # a new view: the buffers start from zero
        state["accum"].zero_()
        state["casts"].zero_()
        state["scene"].render(state["cam"], state["accum"], state["casts"], spp=case["spp"], max_depth=case["depth"],
                              seed=state["seed"])
        return {"accum": state["accum"], "casts": state["casts"]}
    if kind == "batch":
        for accum, casts in state["images"]:
            accum.zero_()
            casts.zero_()
        state["batch"].render(sample_offsets=[0] * case["scenes"])
        return [{"accum": a, "casts": c} for a, c in state["images"]]
    if kind == "guided":
        state["accum"].zero_()
        state["casts"].zero_()
        state["scene"].render_guided(state["guide"], state["cam"], state["accum"], state["casts"], spp=case["spp"],
                                     max_depth=case["depth"], seed=state["seed"], alpha=0.75, train=False,
                                     bounces=case["bounces"], wave_paths=16 * case["width"] * case["height"])
        return {"accum": state["accum"], "casts": state["casts"]}
    if kind == "infer":
        state["guide"].infer(state["pos"], state["nrm"], case["rows"], state["y"])
        return {"y": state["y"]}
    if kind == "train":
        # from given parameters, through the Adam steps, to the trained ones
        n = case["rows"]
        state["guide"].set_params(state["net"])
        for k in range(case["steps"]):
            s = slice(k * n, (k + 1) * n)
            state["guide"].train_step(state["pos"][s], state["nrm"][s], state["sdir"][s], state["weight"][s], n)
        return {"params": state["guide"].params()}
    if kind == "alias":
        state["ctx"].alias_build(state["weights"], case["weights"], state["table"])
        return {"table": state["table"]}
    native.tonemap(state["accum"], case["width"], case["height"], state["rgba"])
    return {"rgba": state["rgba"]}


# ---- work -----------------------------------------------------------------------------


def _ray_flops(tris: int) -> float:
    """A ray that goes straight down an 8-wide tree to one leaf triangle: 8 box
    tests of 13 operations per level, one triangle test of about 70."""
    levels = max(1, math.ceil(math.log(max(tris / 3.0, 1.0)) / math.log(8.0)))
    return 8 * 13 * levels + 70


def _image_work(tris: int, npix: int, spp: int):
    # the image and its casts, read and written; the scene's triangles, once; a
    # camera ray and one light sample's shadow ray per path
    return 40.0 * npix + 36.0 * tris, 2.0 * npix * spp * _ray_flops(tris)


def work(case):
    kind = case["kind"]
    if kind == "trace":
        out = 8 if case["query"] == "closest" else 1
        return {"bytes": (32.0 + out) * case["rays"] + 36.0 * case["tris"],
                "flops": case["rays"] * _ray_flops(case["tris"])}
    if kind == "frame":
        tris = case["tris"] or 1292
        b, f = _image_work(tris, case["width"] * case["height"], case["spp"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        parts = [_image_work(int(t), int(r) ** 2, case["spp"]) for t, r in zip(*_batch_sizes(case))]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    if kind == "guided":
        npix = case["width"] * case["height"]
        b, f = _image_work(case["tris"], npix, case["spp"])
        return {"bytes": b, "flops": f + npix * case["spp"] * 2.0 * sum(i * o for i, o in LAYERS)}
    mac = sum(i * o for i, o in LAYERS)
    params = sum((i + 1) * o for i, o in LAYERS)
    if kind == "infer":
        return {"bytes": case["rows"] * (24.0 + 160.0) + 4.0 * params, "flops": 2.0 * mac * case["rows"]}
    if kind == "train":
        # forward, backward (all layers but the first) and weight gradients;
        # parameters and both moments read and written per step
        per_row = 2.0 * (3 * mac - LAYERS[0][0] * LAYERS[0][1])
        return {"bytes": case["steps"] * (case["rows"] * 40.0 + 24.0 * params),
                "flops": case["steps"] * case["rows"] * per_row}
    if kind == "alias":
        return {"bytes": 24.0 * case["weights"], "flops": 10.0 * case["weights"]}
    n = case["width"] * case["height"]
    return {"bytes": 20.0 * n, "flops": 30.0 * n}


# ---- 64-bit results -------------------------------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind == "trace" and case["query"] == "closest" and case["rays"] * case["tris"] <= 1 << 27:
        return {"t": _exact_t(case, seed), "prim": None}
    if kind == "infer":
        pos, nrm, _, _ = _samples(case, seed)
        net = [p.cpu() for p in _layers(torch.from_numpy(_net(seed)).double())]
        rows = []
        for b in range(0, case["rows"], 1 << 17):
            rows.append(_forward(net, pos[b:b + (1 << 17)].double().cpu(), nrm[b:b + (1 << 17)].double().cpu()))
        return {"y": torch.cat(rows)[:, :40]}
    if kind == "train":
        return {"params": _exact_train(case, seed)}
    return None


def _exact_t(case, seed) -> torch.Tensor:
    """Distance of the closest two-sided hit of every ray, by brute force."""
    soup, _, _, half = _soup(case, seed)
    rays = _rays(case, seed, half).double().cpu()
    tri = torch.from_numpy(soup).double().reshape(-1, 3, 3)
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    out = []
    step = max(1, (1 << 22) // len(soup))
    for b in range(0, len(rays), step):
        o, tmax, d = rays[b:b + step, None, 0:3], rays[b:b + step, 3], rays[b:b + step, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, len(tri), 3), e2.expand(len(o), -1, 3))
        det = (p * e1).sum(-1)
        s = o - a
        q = torch.linalg.cross(s, e1.expand(len(o), -1, 3))
        u, v, t = (s * p).sum(-1) / det, (d * q).sum(-1) / det, (e2 * q).sum(-1) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0) & (t <= tmax[:, None])
        out.append(torch.where(ok, t, torch.full_like(t, math.inf)).amin(1))
    return torch.cat(out)


def _layers(params: torch.Tensor) -> list:
    """Weight [out, in] and bias of each layer, as views of the parameters."""
    at, net = 0, []
    for fan_in, fan_out in LAYERS:
        net.append(params[at:at + fan_in * fan_out].view(fan_out, fan_in))
        net.append(params[at + fan_in * fan_out:at + (fan_in + 1) * fan_out])
        at += (fan_in + 1) * fan_out
    return net


def _forward(net, pos, nrm) -> torch.Tensor:
    x = (pos / 50.0).clamp(-1.0, 1.0)
    angle = math.pi * x[:, :, None] * (2.0 ** torch.arange(12, dtype=torch.float64))
    enc = torch.stack([torch.sin(angle), torch.cos(angle)], dim=-1).reshape(len(x), 72)
    h = torch.cat([enc, nrm, torch.zeros(len(x), 5, dtype=torch.float64)], dim=1)
    for l in range(5):
        h = h @ net[2 * l].T + net[2 * l + 1]
        if l < 4:
            h = torch.relu(h)
    return h


def _log_density(y, w) -> torch.Tensor:
    """Log density of the von Mises-Fisher mixture of network outputs y at w."""
    lobe = y[:, :40].reshape(-1, 8, 5)
    k = torch.exp(lobe[..., 1].clamp(-4.0, 7.0))
    mu = torch.nn.functional.normalize(lobe[..., 2:5], dim=-1)
    log_norm = torch.log(k) - math.log(2.0 * math.pi) - torch.log1p(-torch.exp(-2.0 * k))
    c = (mu * w[:, None, :]).sum(-1)
    return torch.logsumexp(torch.log_softmax(lobe[..., 0], dim=1) + log_norm + k * (c - 1.0), dim=1)


def _exact_train(case, seed) -> torch.Tensor:
    """The parameters after the case's Adam steps."""
    pos, nrm, sdir, weight = (t.double().cpu() for t in _samples(case, seed))
    params = torch.from_numpy(_net(seed)).double()
    m, v = torch.zeros_like(params), torch.zeros_like(params)
    n = case["rows"]
    for k in range(case["steps"]):
        s = slice(k * n, (k + 1) * n)
        p = params.clone().requires_grad_(True)
        net = _layers(p)
        c = weight[s] / weight[s].mean()
        grad = torch.zeros_like(params)
        for b in range(0, n, 16384):
            r = slice(k * n + b, min(k * n + b + 16384, (k + 1) * n))
            loss = -(c[b:b + 16384] * _log_density(_forward(net, pos[r], nrm[r]), sdir[r])).sum() / n
            grad += torch.autograd.grad(loss, p, retain_graph=False)[0]
            net = _layers(p)
        m = 0.9 * m + 0.1 * grad
        v = 0.999 * v + 0.001 * grad * grad
        t = k + 1
        params = params - 1e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return params
