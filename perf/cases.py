"""Workloads of this framework as its users run them, for timing one build against another.

A case is one call (or the few calls of one frame) through the public entry points: rays traced
against a built structure, a frame of the path tracer, a query of the radiance cache, a training step.
The scenes are the package's own (kiraray_gb300/scenes.py) at the sizes of its configurations; the
seed of a case places the camera, draws the rays and picks the sample streams, the records and the
targets.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from kiraray_gb300 import scenes
from kiraray_gb300.accel import Accel
from kiraray_gb300.convergence import Accumulator, tonemap
from kiraray_gb300.nrc import NeuralRadianceCache
from kiraray_gb300.wavefront import WavefrontPathTracer

FULL_GRID, FULL_SPHERES = 2048, 500     # the 10.9M-triangle scene


def listed() -> list:
    return [
        # The closest-hit query that a renderer makes for every pixel: camera rays of a full frame.
        dict(name="camera rays 1080p", kind="rays", scene="large", set="camera", grid=FULL_GRID,
             spheres=FULL_SPHERES, width=1920, height=1080, levels=1),
        # The same after one diffuse bounce: every ray goes its own way.
        dict(name="bounce rays 1080p", kind="rays", scene="large", set="bounce", grid=FULL_GRID,
             spheres=FULL_SPHERES, width=1920, height=1080, levels=1),
        # Light visibility from every pixel's hit point (any hit, bounded rays).
        dict(name="shadow rays 1080p", kind="rays", scene="large", set="shadow", grid=FULL_GRID,
             spheres=FULL_SPHERES, width=1920, height=1080, levels=1),
        # Picking and probing: about a thousand rays against a small scene, where latency counts.
        dict(name="probe rays", kind="rays", scene="cornell", set="bounce", grid=0, spheres=0, width=41,
             height=27, levels=1),
        # An animated scene: new instance transforms, then a preview's camera rays over two levels.
        dict(name="moving instances 960x540", kind="rays", scene="large", set="camera", grid=FULL_GRID,
             spheres=FULL_SPHERES, width=960, height=540, levels=2),
        # One sample per pixel of the large scene at full resolution, surfaces only.
        dict(name="frame large 1080p", kind="frame", scene="large", grid=FULL_GRID, spheres=FULL_SPHERES,
             width=1920, height=1080, depth=8, views=1, spp=1, cache=False, display=False),
        # One sample per pixel of the Cornell box.
        dict(name="frame cornell 512", kind="frame", scene="cornell", grid=0, spheres=0, width=512,
             height=512, depth=5, views=1, spp=1, cache=False, display=False),
        # One sample per pixel through a heterogeneous medium.
        dict(name="frame volume 1024", kind="frame", scene="volume", grid=256, spheres=0, width=1024,
             height=1024, depth=16, views=1, spp=1, cache=False, display=False),
        # A viewer's progressive preview: a small frame, added up and tone-mapped for display.
        dict(name="viewer 241x135", kind="frame", scene="large", grid=FULL_GRID, spheres=FULL_SPHERES,
             width=241, height=135, depth=8, views=1, spp=1, cache=False, display=True),
        # Batched views with the radiance cache answering and training online.
        dict(name="cached views 8x480x270", kind="frame", scene="large", grid=FULL_GRID,
             spheres=FULL_SPHERES, width=480, height=270, depth=8, views=8, spp=1, cache=True,
             display=False),
        # The cache asked for a frame's worth of path vertices.
        dict(name="cache query 1.5M", kind="query", records=1500001, log2_table=19, hidden=5),
        # One optimiser step on a full training batch, and the answers of the updated cache.
        dict(name="cache train 64k", kind="train", records=65536, log2_table=19, hidden=5),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["rays", "rays", "rays2", "frame", "frame", "volume", "cached", "query", "train"])
    if kind in ("rays", "rays2"):
        h = _log_int(rng, 9, 1080)
        small = kind == "rays" and rng.random() < 0.2
        return dict(kind="rays", scene="cornell" if small else "large",
                    set="camera" if kind == "rays2" else rng.choice(["camera", "bounce", "shadow"]),
                    grid=0 if small else _log_int(rng, 65, FULL_GRID),
                    spheres=0 if small else rng.randint(1, FULL_SPHERES),
                    width=max(1, min(1920, int(h * rng.uniform(0.8, 1.9)))), height=h,
                    levels=2 if kind == "rays2" else 1)
    if kind in ("frame", "cached"):
        cached = kind == "cached"
        h = _log_int(rng, 40, 540 if cached else 1080)
        big = cached or rng.random() < 0.7
        return dict(kind="frame", scene="large" if big else "cornell",
                    grid=_log_int(rng, 129, FULL_GRID) if big else 0,
                    spheres=rng.randint(1, FULL_SPHERES) if big else 0,
                    width=max(8, min(1920, int(h * rng.uniform(0.8, 1.9)))), height=h,
                    depth=rng.randint(2, 8), views=rng.randint(1, 4) if cached else 1,
                    spp=1 if cached or h > 270 else rng.randint(1, 2), cache=cached,
                    display=not cached and rng.random() < 0.5)
    if kind == "volume":
        h = _log_int(rng, 48, 1024)
        return dict(kind="frame", scene="volume", grid=rng.choice([64, 128, 256]), spheres=0,
                    width=max(16, min(1024, int(h * rng.uniform(0.7, 1.0)))), height=h,
                    depth=rng.randint(4, 16), views=1, spp=1, cache=False, display=False)
    hidden = rng.randint(2, 5)
    if kind == "query":
        return dict(kind="query", records=_log_int(rng, 100, 1500000), log2_table=rng.randint(14, 19),
                    hidden=hidden)
    return dict(kind="train", records=_log_int(rng, 500, 65536), log2_table=rng.randint(12, 19),
                hidden=hidden)


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=6)
def _scene(kind: str, grid: int, spheres: int):
    """A scene of the package; the host arrays are kept between cases, as a program keeps its assets."""
    if kind == "large":
        return scenes.large_scene(64, 64, grid=grid, n_spheres=spheres)
    if kind == "volume":
        return scenes.volume_box(64, 64, grid=grid)
    return scenes.cornell_box(64, 64)


@functools.lru_cache(maxsize=2)
def _world_triangles(kind: str, grid: int, spheres: int) -> np.ndarray:
    return _scene(kind, grid, spheres).world_triangles()


def _camera(kind: str, width: int, height: int, seed: int, k: int = 0):
    """The scene's camera, turned up to ten degrees around the scene by the seed."""
    a = math.radians(np.random.default_rng([seed, k]).uniform(-10, 10))
    if kind == "large":
        return scenes._camera((62.0 * math.sin(a), 22.0, -62.0 * math.cos(a)), (0.0, 2.0, 0.0), 45.0,
                              width, height)
    return scenes._camera((0.5 + 1.9 * math.sin(a), 0.5, 0.5 - 1.9 * math.cos(a)), (0.5, 0.5, 0.0), 40.0,
                          width, height)


def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _camera_rays(cam, width: int, height: int, gen) -> torch.Tensor:
    """Rays through jittered pixels, row-major, float32 [height * width, 8]."""
    n = width * height
    i = torch.arange(n, device="cuda")
    u = torch.rand((n, 2), generator=gen, device="cuda", dtype=torch.float64)
    x = 2 * ((i % width) + u[:, 0]) / width - 1
    y = 1 - 2 * ((i // width) + u[:, 1]) / height
    t = cam.film_size[1] * 0.5 / cam.focal_length
    d = torch.stack([t * cam.aspect_ratio * x, t * y, -torch.ones_like(x)], -1)
    d = d / d.norm(dim=-1, keepdim=True) @ torch.tensor(np.asarray(cam.rotation, np.float64).T, device="cuda")
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, :3] = torch.tensor(cam.position, dtype=torch.float32, device="cuda")
    rays[:, 4:7] = d.float()
    rays[:, 7] = math.inf
    return rays


def _secondary_rays(tris: np.ndarray, rays, hits, which: str, scene_kind: str, gen) -> torch.Tensor:
    """From the hit points of `rays`: cosine-weighted bounces, or bounded rays to points of the lights.
    As many as `rays`, in their order: the hit points stand in for the rays that missed."""
    prim = hits.view(torch.int32)[:, 3].to(torch.int64)
    found = (prim >= 0).nonzero()[:, 0]
    if found.numel() == 0:
        return rays
    n_rays = rays.shape[0]
    ok = found[torch.arange(n_rays, device="cuda") * found.numel() // n_rays]
    v = torch.from_numpy(tris).cuda()[prim[ok]].reshape(-1, 3, 3).double()
    d0 = rays[ok, 4:7].double()
    p = rays[ok, :3].double() + hits[ok, :1].double() * d0
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n = n / (n.norm(dim=-1, keepdim=True) + 1e-30)
    n = torch.where((n * d0).sum(-1, keepdim=True) > 0, -n, n)
    m = p.shape[0]
    u = torch.rand((m, 3), generator=gen, device="cuda", dtype=torch.float64)
    out = torch.zeros((m, 8), device="cuda")
    o = p + n * 1e-4
    if which == "shadow":
        if scene_kind == "large":       # four 4x4 quads at y = 30
            q = (u[:, 0] * 4).floor()
            to = torch.stack([(q % 2) * 40 - 20 + 4 * u[:, 1] - 2, torch.full_like(q, 29.99),
                              (q // 2).floor() * 40 - 20 + 4 * u[:, 2] - 2], -1)
        else:
            to = torch.stack([0.375 + 0.25 * u[:, 0], torch.full_like(u[:, 0], 0.9985),
                              0.375 + 0.25 * u[:, 1]], -1)
        out[:, 4:7], out[:, 7] = (to - o).float(), 1.0
    else:
        r, phi = u[:, 0].sqrt(), 2 * math.pi * u[:, 1]
        a = torch.zeros_like(n)
        big = n[:, 0].abs() > 0.9
        a[big, 1], a[~big, 0] = 1.0, 1.0
        t = torch.linalg.cross(a, n)
        t = t / t.norm(dim=-1, keepdim=True)
        b = torch.linalg.cross(n, t)
        w = (1 - u[:, 0]).clamp_min(0).sqrt()
        out[:, 4:7] = ((r * phi.cos())[:, None] * t + (r * phi.sin())[:, None] * b + w[:, None] * n).float()
        out[:, 7] = math.inf
    out[:, :3] = o.float()
    return out.contiguous()


def _geometries(sc):
    """Each mesh's object-space triangles once, and the instances over them."""
    geoms, key_of, inst = [], {}, []
    for mi, xf in sc.instances:
        m = sc.meshes[mi]
        key = (id(m.positions), id(m.indices))
        if key not in key_of:
            key_of[key] = len(geoms)
            geoms.append(np.asarray(m.positions, np.float32)[np.asarray(m.indices)].reshape(-1, 9))
        inst.append((key_of[key], np.asarray(xf, np.float32)))
    return geoms, inst


# --------------------------------------------------------------- the cache
_PRIMES = (1, 2654435761, 805459861)
_LEVELS, _BASE, _TOP, _BINS = 16, 16, 2048, 4


def _levels(log2_table: int) -> list:
    """(cells per axis, first entry, entries, dense) of every level of the hash grid."""
    b = math.exp((math.log(_TOP) - math.log(_BASE)) / (_LEVELS - 1))
    out, off = [], 0
    for k in range(_LEVELS):
        res = int(math.floor(_BASE * b ** k + 1e-6))
        dense = (res + 1) ** 3 <= 1 << log2_table
        size = (res + 1) ** 3 if dense else 1 << log2_table
        out.append((res, off, size, dense))
        off += size
    return out


def _parameters(case: dict, seed: int):
    """Weights and hash table of a cache that has been trained for a while: the table's features are
    of the order of a tenth, the layers keep their inputs' scale."""
    rng = np.random.default_rng(seed)
    n_table = sum(lv[2] for lv in _levels(case["log2_table"])) * 2
    table = (rng.random(n_table, dtype=np.float32) - np.float32(0.5)) * np.float32(0.6)
    ws = []
    for k in range(case["hidden"] + 1):
        rows, used = (64, 64) if k < case["hidden"] else (16, 3)
        fan_in = 2 * _LEVELS + 5 * _BINS + 3 if k == 0 else 64
        w = np.zeros((rows, 64), np.float32)
        w[:used, :fan_in] = (rng.random((used, fan_in), dtype=np.float32) * 2 - 1) * math.sqrt(6.0 / fan_in)
        ws.append(w)
    return ws, table


def _records(n: int, seed: int) -> torch.Tensor:
    """Path vertices as a frame's pixels give them: neighbours in the list lie near each other on a
    surface, a bounce apart."""
    g = _generator(seed)
    side = max(1, int(math.sqrt(n)))
    i = torch.arange(n, device="cuda")
    x = torch.stack([(i % side).float() / side, (i // side).float() / (n / side)], -1)
    x = (x + 0.05 * torch.randn((n, 2), generator=g, device="cuda")).clamp(0, 1)
    y = 0.3 + 0.1 * torch.sin(9 * x[:, 0]) * torch.cos(7 * x[:, 1])
    unit = torch.randn((n, 2, 3), generator=g, device="cuda")
    unit[:, :, 1] = unit[:, :, 1].abs()
    unit = unit / unit.norm(dim=-1, keepdim=True)
    rest = torch.rand((n, 4), generator=g, device="cuda")
    pos = torch.stack([x[:, 0], y, x[:, 1]], -1) * 100 - 50
    return torch.cat([pos, unit[:, 0], rest[:, :1], rest[:, 1:], unit[:, 1]], -1).contiguous()


def _targets(records: torch.Tensor, seed: int) -> torch.Tensor:
    """Noisy one-sample radiance that varies over the surface and with the albedo."""
    p = records[:, :3] / 50
    base = 0.5 + 0.4 * torch.sin(5 * p[:, :1]) * torch.cos(4 * p[:, 2:3])
    noise = torch.rand((records.shape[0], 1), generator=_generator(seed + 1), device="cuda")
    return (base * records[:, 7:10] * (0.25 + 1.5 * noise)).contiguous()


def _predict64(case: dict, seed: int) -> torch.Tensor:
    """The cache's answers in 64 bits: trilinear hash-grid features, one-blob inputs, the layers."""
    rec = _records(case["records"], seed).double()
    ws, table = _parameters(case, seed)
    tab = torch.from_numpy(table).cuda().double().reshape(-1, 2)
    p = ((rec[:, :3] + 50) / 100).clamp(0, 1)
    feats = []
    for res, off, size, dense in _levels(case["log2_table"]):
        s = p * res
        base = s.floor().clamp(0, res - 1)
        fr = (s - base).clamp(0, 1)
        base = base.to(torch.int64)
        f = torch.zeros((rec.shape[0], 2), dtype=torch.float64, device="cuda")
        for k in range(8):
            bit = [k & 1, k >> 1 & 1, k >> 2 & 1]
            c = [base[:, a] + bit[a] for a in range(3)]
            if dense:
                idx = c[0] + (res + 1) * (c[1] + (res + 1) * c[2])
            else:
                idx = (c[0] ^ (c[1] * _PRIMES[1]) ^ (c[2] * _PRIMES[2])) & (size - 1)
            w = torch.ones_like(fr[:, 0])
            for a in range(3):
                w = w * (fr[:, a] if bit[a] else 1 - fr[:, a])
            f += w[:, None] * tab[off + idx]
        feats.append(f)
    centre = (torch.arange(_BINS, device="cuda") + 0.5) / _BINS

    def blob(v):
        return torch.exp(-0.5 * ((v[:, None] - centre) * _BINS) ** 2)

    for o in (3, 10):
        feats.append(blob(torch.acos(rec[:, o + 2].clamp(-1, 1)) / math.pi))
        feats.append(blob(torch.atan2(rec[:, o + 1], rec[:, o]) / (2 * math.pi) + 0.5))
    feats += [blob(1 - torch.exp(-rec[:, 6])), rec[:, 7:10]]
    x = torch.cat(feats, -1)
    x = torch.nn.functional.pad(x, (0, 64 - x.shape[1]))
    for k, w in enumerate(ws):
        x = x @ torch.from_numpy(w).cuda().double().T
        if k < case["hidden"]:
            x = x.clamp_min(0)
    return x[:, :3].contiguous()


# -------------------------------------------------------- state and passes
def _prepare_rays(case: dict, seed: int) -> dict:
    sc = _scene(case["scene"], case["grid"], case["spheres"])
    gen = _generator(seed)
    cam = _camera(case["scene"], case["width"], case["height"], seed)
    rays = _camera_rays(cam, case["width"], case["height"], gen)
    if case["levels"] == 2:
        geoms, inst = _geometries(sc)
        acc = Accel.instanced(geoms, inst)
        moved = np.stack([xf for _, xf in inst])
        shift = np.random.default_rng(seed).uniform(-0.5, 0.5, (moved.shape[0], 3)).astype(np.float32)
        moved[1:, :, 3] += shift[1:]                     # the terrain stays
    else:
        tris = _world_triangles(case["scene"], case["grid"], case["spheres"])
        acc, moved = Accel(tris), None
        if case["set"] != "camera":
            rays = _secondary_rays(tris, rays, acc.trace_closest(rays), case["set"], case["scene"], gen)
    n, any_hit = rays.shape[0], case["set"] == "shadow"
    out = torch.empty(n, dtype=torch.uint8, device="cuda") if any_hit else torch.empty((n, 4), device="cuda")
    # a hit is t, two barycentrics and the triangle's id
    hits = None if any_hit else {"t": out[:, 0], "b": out[:, 1:3], "prim": out.view(torch.int32)[:, 3]}
    return dict(kind="rays", accel=acc, rays=rays, out=out, hits=hits, any_hit=any_hit, moved=moved)


def _run_rays(s: dict):
    if s["moved"] is not None:
        s["accel"].update_instances(s["moved"])
    if s["any_hit"]:
        return s["accel"].trace_any(s["rays"], s["out"])
    s["accel"].trace_closest(s["rays"], s["out"])
    return s["hits"]


def _prepare_frame(case: dict, seed: int) -> dict:
    sc = _scene(case["scene"], case["grid"], case["spheres"])
    w, h = case["width"], case["height"]
    pt = WavefrontPathTracer({"max_depth": case["depth"]}, spp=case["spp"], seed=seed % 100000)
    pt.set_scene(sc)
    s = dict(kind="frame", pass_=pt, frame=0, views=None, cache=None, acc=None)
    if case["views"] > 1 or case["cache"]:
        s["views"] = [(_camera(case["scene"], w, h, seed, k), w, h, seed % 100000 + 1000 * k)
                      for k in range(case["views"])]
        pt.resize_views(s["views"])
        s["out"] = torch.empty((pt.n_pixels, 4), device="cuda")
    else:
        s["camera"] = _camera(case["scene"], w, h, seed)
        pt.resize(w, h)
        s["out"] = torch.empty((h, w, 4), device="cuda")
    if case["cache"]:
        lo, hi = pt.cache_box()
        s["cache"] = NeuralRadianceCache(lo, hi, seed=3, epsilon=1e-8)
        pt.set_nrc(s["cache"], train=True)
    if case["display"]:
        s["acc"], s["shown"] = Accumulator(w, h), torch.empty((h, w, 4), device="cuda")
    return s


def _run_frame(s: dict):
    s["frame"] += 1
    pt = s["pass_"]
    if s["views"] is not None:
        pt.begin_frame_views(s["frame"], s["views"])
        out = {"frame": pt.render_flat(s["out"])}
    else:
        pt.begin_frame(s["frame"], s["camera"])
        out = {"frame": pt.render(s["out"])}
    if s["cache"] is not None:
        out["weights"] = s["cache"].params(0)
    if s["acc"] is not None:
        s["acc"].add(out["frame"])
        out["sum"] = s["acc"].sum
        out["shown"] = tonemap(out["frame"], "aces", 1.0, True, s["shown"])
    return out


def _prepare_cache(case: dict, seed: int) -> dict:
    cache = NeuralRadianceCache((-50, -50, -50), (50, 50, 50), seed=3, log2_table_size=case["log2_table"],
                                hidden_layers=case["hidden"], epsilon=1e-8)
    ws, table = _parameters(case, seed)
    cache.set_params(0, np.concatenate([w.reshape(-1) for w in ws]))
    cache.set_params(1, table)
    rec = _records(case["records"], seed)
    s = dict(kind=case["kind"], cache=cache, records=rec)
    if case["kind"] == "train":
        s["targets"] = _targets(rec, seed)
        s["whole"] = case["log2_table"] <= 14
    return s


def _run_train(s: dict):
    loss = s["cache"].train_step(s["records"], s["targets"])
    out = {"loss": float(loss), "weights": s["cache"].params(0),
           "predictions": s["cache"].query(s["records"])}
    if s["whole"]:
        out["table"] = s["cache"].params(1)
    return out


def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "rays":
        return _prepare_rays(case, seed)
    if case["kind"] == "frame":
        return _prepare_frame(case, seed)
    return _prepare_cache(case, seed)


def run(state: dict):
    if state["kind"] == "rays":
        return _run_rays(state)
    if state["kind"] == "frame":
        return _run_frame(state)
    if state["kind"] == "query":
        return state["cache"].query(state["records"])
    return _run_train(state)


# ------------------------------------------------------------ what it takes
def work(case: dict) -> dict:
    """Bytes: inputs read once and outputs written once.  Operations: eight slab tests (12 operations
    each) for every level of an eight-wide tree over the triangles and one triangle test (60) a ray; a
    path counts a closest-hit ray and a light ray for each of its vertices (0.8^k of the paths reach
    vertex k); the cache's layers, three times for a training step."""
    if case["kind"] in ("query", "train"):
        n, layers = case["records"], 2 * 64 * 64 * case["hidden"] + 2 * 64 * 3
        entries = sum(lv[2] for lv in _levels(case["log2_table"]))
        table = min(n * _LEVELS * 8, entries) * 4
        if case["kind"] == "query":
            return {"bytes": n * (52 + 12) + table, "flops": n * layers}
        params = 2 * min(n * _LEVELS * 8, entries) + 64 * 64 * case["hidden"] + 64 * 16
        return {"bytes": n * (52 + 12 + 12) + params * (3 * 4 * 2 + 2), "flops": 4 * n * layers}
    tris = 36 if case["scene"] != "large" else 2 * (case["grid"] - 1) ** 2 + 5120 * case["spheres"] + 8
    per_ray = 96 * max(1.0, math.log(tris, 8)) + 60
    pixels = case["width"] * case["height"]
    if case["kind"] == "rays":
        return {"bytes": pixels * (32 + (1 if case["set"] == "shadow" else 16)), "flops": pixels * per_ray}
    paths = pixels * case["views"] * case["spp"]
    rays = paths * 2 * sum(0.8 ** k for k in range(case["depth"] + 1))
    return {"bytes": pixels * case["views"] * 16 * (4 if case["display"] else 1), "flops": rays * per_ray}


def exact(case: dict, seed: int):
    """64-bit answers: the cache's predictions, and the hits of rays in the small scene (every triangle
    tested).  Frames, and rays in the large scene, have none that is quick to compute."""
    if case["kind"] == "query":
        return _predict64(case, seed)
    if case["kind"] != "rays" or case["scene"] != "cornell" or case["set"] == "shadow":
        return None
    rays = _prepare_rays(case, seed)["rays"].double()
    v = torch.from_numpy(_world_triangles("cornell", 0, 0)).cuda().double().reshape(-1, 3, 3)
    o, d = rays[:, None, :3], rays[:, None, 4:7]
    e1, e2 = v[None, :, 1] - v[None, :, 0], v[None, :, 2] - v[None, :, 0]
    best_t = torch.full((rays.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    best_b = torch.zeros((rays.shape[0], 2), dtype=torch.float64, device="cuda")
    for k in range(0, rays.shape[0], 1 << 16):
        c = slice(k, k + (1 << 16))
        h = torch.linalg.cross(d[c].expand(-1, e2.shape[1], -1), e2.expand(d[c].shape[0], -1, -1))
        det = (e1 * h).sum(-1)
        s = o[c] - v[None, :, 0]
        b1 = (s * h).sum(-1) / det
        q = torch.linalg.cross(s, e1.expand(s.shape[0], -1, -1))
        b2 = (d[c] * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        ok = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t > 0) & (det != 0)
        t = torch.where(ok, t, torch.inf)
        tt, i = t.min(1)
        best_t[c] = tt
        hit = torch.isfinite(tt)
        b = torch.stack([b1.gather(1, i[:, None])[:, 0], b2.gather(1, i[:, None])[:, 0]], -1)
        best_b[c] = torch.where(hit[:, None], b, 0.0)
    return {"t": best_t, "b": best_b, "prim": None}
