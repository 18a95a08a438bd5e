"""The work that programs have this library do, as cases that can be timed: ray
queries from device and host memory, tree builds, path-traced frames, a batch of
scenes, and the path-guiding network, from the smallest calls to the largest.

A case is a dict of plain values. Its "kind" names the call:
  rays    bbg_intersect / bbg_intersect_any over device-resident rays
  host    a closest-hit and an any-hit batch submitted from page-locked host
          memory and waited for once
  build   an acceleration structure built on the device, first rays traced
          through it, and released
  frame   a rendered frame (host or device film)
  batch   several small scenes rendered as one wavefront
  train   the guiding network's forward and backward pass over a batch
Scenes and rays are those of bulbit_b200.scenes, seeded by the case's seed.
"""
import math

import numpy as np
import torch

from bulbit_b200 import abi, lib, scenes


def listed():
    return [
        # A few picking or probe rays against a small mesh: latency of one call.
        {"name": "rays_1k", "kind": "rays", "query": "closest", "scene": "soup", "size": 20_000, "n": 1024},
        # A ragged batch of short occlusion rays (ambient occlusion) in a mesh scene.
        {"name": "ao_cornell", "kind": "rays", "query": "any", "scene": "cornell", "size": 7, "n": 2_000_003},
        # Ray throughput: incoherent closest-hit rays through a million triangles.
        {"name": "rays_4m_soup1m", "kind": "rays", "query": "closest", "scene": "soup", "size": 1 << 20, "n": 1 << 22},
        # A program with its rays in host memory: both queries of a step in flight.
        {"name": "host_pair_1m", "kind": "host", "scene": "soup", "size": 1 << 18, "n": 1_000_003},
        # A changed mesh: the reference's SAH tree rebuilt on the device.
        {"name": "build_sah_1m", "kind": "build", "method": "sah", "scene": "soup", "size": 1 << 20, "n": 65_536},
        # A static mesh worth a better tree: references split on the device.
        {"name": "build_split_300k", "kind": "build", "method": "split", "scene": "cornell", "size": 7, "n": 65_536},
        # The README example: spheres, spot and infinite light, host film.
        {"name": "frame_readme", "kind": "frame", "scene": "readme", "size": 0, "width": 320, "height": 180, "spp": 16,
         "bounces": 8, "material": "diffuse", "film": "host", "wave": 0, "strata": 0, "filter": 0, "guided": False},
        # A preview frame of odd size: glass sphere, stratified samples, Gaussian filter.
        {"name": "frame_glass_preview", "kind": "frame", "scene": "cornell", "size": 6, "width": 501, "height": 333,
         "spp": 16, "bounces": 16, "material": "glass", "film": "host", "wave": 0, "strata": 4,
         "filter": abi.BBG_FILTER_GAUSSIAN, "guided": False},
        # The path-tracing benchmark frame: 1,310,734 triangles, 2^26 paths in one wave.
        {"name": "frame_cornell_1024", "kind": "frame", "scene": "cornell", "size": 8, "width": 1024, "height": 1024,
         "spp": 64, "bounces": 16, "material": "gold", "film": "device", "wave": 1 << 26, "strata": 0, "filter": 0,
         "guided": False},
        # A guided frame (fixed guide): network inference between two shading passes.
        {"name": "frame_guided_256", "kind": "frame", "scene": "cornell", "size": 6, "width": 256, "height": 256,
         "spp": 16, "bounces": 12, "material": "gold", "film": "host", "wave": 0, "strata": 0, "filter": 0,
         "guided": True},
        # Thumbnails of a set of scenes, each too small to fill the GPU by itself.
        {"name": "batch_8x96", "kind": "batch", "scenes": 8, "width": 96, "height": 96, "spp": 32, "bounces": 12},
        # One training batch of the guide at its default size.
        {"name": "train_64k", "kind": "train", "n": 1 << 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "host", "build", "build", "frame", "frame", "frame", "batch", "train"])
    scene = rng.choice(["soup", "cornell"])
    size = _log_int(rng, 1000, 1 << 20) if scene == "soup" else rng.randint(2, 8)
    if kind == "rays":
        return {"kind": kind, "query": rng.choice(["closest", "any"]), "scene": scene, "size": size,
                "n": _log_int(rng, 500, 1 << 22)}
    if kind == "host":
        return {"kind": kind, "scene": scene, "size": size, "n": _log_int(rng, 1000, 3_000_000)}
    if kind == "build":
        method = rng.choice(["sah", "split", "linear"])
        if method == "split" and scene == "soup":
            size = min(size, 1 << 18)
        return {"kind": kind, "method": method, "scene": scene, "size": size, "n": _log_int(rng, 1000, 200_000)}
    if kind == "frame":
        scene = rng.choice(["readme", "cornell", "cornell", "cornell"])
        strata = rng.choice([0, 0, 2, 4])
        spp = strata * rng.randint(1, 8) if strata else _log_int(rng, 1, 64)
        guided = scene == "cornell" and rng.random() < 0.25
        return {"kind": kind, "scene": scene, "size": 0 if scene == "readme" else rng.randint(3, 8),
                "width": _log_int(rng, 40, 640), "height": _log_int(rng, 40, 640), "spp": spp,
                "bounces": rng.randint(1, 20),
                "material": rng.choice(["diffuse", "gold", "glass", "rough_glass", "metal"]) if scene != "readme" else "diffuse",
                "film": rng.choice(["host", "device"]), "wave": 0, "strata": 0 if guided else strata,
                "filter": rng.choice([abi.BBG_FILTER_BOX, abi.BBG_FILTER_TENT, abi.BBG_FILTER_GAUSSIAN]),
                "guided": guided}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 16), "width": _log_int(rng, 32, 160),
                "height": _log_int(rng, 32, 160), "spp": _log_int(rng, 2, 32), "bounces": rng.randint(2, 16)}
    return {"kind": "train", "n": _log_int(rng, 1000, 1 << 17)}


# ------------------------------------------------------------------ inputs

def _material(name):
    return {"diffuse": lambda: scenes.diffuse((0.6, 0.5, 0.4)),
            "gold": lambda: None,  # the scene's own rough gold conductor
            "glass": lambda: scenes.dielectric(1.5),
            "rough_glass": lambda: scenes.dielectric(1.5, roughness=0.3),
            "metal": lambda: scenes.metallic_roughness((0.8, 0.6, 0.3), 0.7, 0.4)}[name]()


def _geometry(case, seed):
    if case["scene"] == "soup":
        return scenes.triangle_soup(case["size"], seed=seed)
    return scenes.cornell_icosphere(levels=case["size"], seed=seed)


def _rays(case, seed):
    """(closest, any) ray sets: toward the soup's cube from outside it, or from
    points inside the box in uniform directions (any-hit rays of length 0.5)."""
    n = case["n"]
    if case["scene"] == "soup":
        return scenes.soup_rays(n, seed=seed)
    g = np.random.default_rng(seed)
    d = g.standard_normal((n, 3), dtype=np.float32)
    closest = np.empty((n, 8), np.float32)
    closest[:, 0:3] = g.random((n, 3), dtype=np.float32) * np.float32(1.9) - np.float32(0.95)
    closest[:, 3:6] = d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), np.float32(1e-6))
    closest[:, 6] = 1e-4
    closest[:, 7] = np.inf
    short = closest.copy()
    short[:, 7] = 0.5
    return closest, short


GUIDE_AABB = (-1.0, -1.0, -1.0, 1.0, 1.0, 1.0)
GUIDE_SHAPES = ((64, 80), (64,), (64, 64), (64,), (64, 64), (64,), (40, 64), (40,))


def _guide_params(seed):
    """A guide part-way through training: every weight at its initial scale, the
    eight lobes about the cube's diagonals."""
    g = np.random.default_rng(seed)
    parts = []
    for s in GUIDE_SHAPES:
        if len(s) == 2:
            a = math.sqrt(6.0 / (s[0] + s[1])) if s[0] == 64 else 0.1
            parts.append(g.uniform(-a, a, s))
        else:
            parts.append(g.uniform(-0.05, 0.05, s))
    lobes = parts[-1].reshape(8, 5)
    for j in range(8):
        lobes[j, 1:4] += [1.0 if j & 1 else -1.0, 1.0 if j & 2 else -1.0, 1.0 if j & 4 else -1.0]
        lobes[j, 4] += math.log(3.0)
    return np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _training_batch(n, seed):
    """Queries (position, normal, outgoing direction, roughness), directions, weights."""
    g = np.random.default_rng(seed + 1)

    def unit():
        v = g.standard_normal((n, 3)).astype(np.float32)
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    raw = np.empty((n, 10), np.float32)
    raw[:, 0:3] = g.uniform(-1, 1, (n, 3))
    raw[:, 3:6] = unit()
    raw[:, 6:9] = unit()
    raw[:, 9] = g.uniform(0.05, 1.0, n)
    return raw, unit(), g.exponential(1.0, n).astype(np.float32)


def _frame_scene(case, seed):
    if case["scene"] == "readme":
        s = scenes.readme_sphere(case["width"], case["height"], case["spp"], case["bounces"])
    else:
        s = scenes.cornell_icosphere(levels=case["size"], width=case["width"], height=case["height"], spp=case["spp"],
                                     max_bounces=case["bounces"], seed=seed, sphere_material=_material(case["material"]))
    s.seed = seed
    s.camera.filter_type = case["filter"]
    if case["filter"] != abi.BBG_FILTER_BOX:
        s.camera.filter_extent = 2.0
    return s


def prepare(case, seed):
    state = {"case": case}
    kind = case["kind"]
    if kind in ("rays", "host"):
        state["accel"] = lib.GpuAccel(_geometry(case, seed), device_sah=True)
        closest, short = _rays(case, seed + 1)
        if kind == "rays":
            state["rays"] = torch.from_numpy(closest if case["query"] == "closest" else short).cuda()
            state["out"] = (torch.empty((case["n"], 4), dtype=torch.float32, device="cuda") if case["query"] == "closest"
                            else torch.empty(case["n"], dtype=torch.uint8, device="cuda"))
        else:
            state["closest"] = torch.from_numpy(closest).pin_memory()
            state["any"] = torch.from_numpy(short).pin_memory()
            state["hits"] = torch.empty((case["n"], 4), dtype=torch.float32, pin_memory=True)
            state["occluded"] = torch.empty(case["n"], dtype=torch.uint8, pin_memory=True)
    elif kind == "build":
        state["scene"] = _geometry(case, seed)
        state["rays"] = torch.from_numpy(_rays(case, seed + 1)[0]).cuda()
        state["out"] = torch.empty((case["n"], 4), dtype=torch.float32, device="cuda")
    elif kind == "frame":
        s = _frame_scene(case, seed)
        state["accel"] = lib.GpuAccel(s, device_sah=True)
        state["integrator"] = lib.GpuPathIntegrator(state["accel"], s)
        if case["guided"]:
            state["guide"] = lib.GpuGuide(GUIDE_AABB, seed=1)
            state["guide"].set_params(_guide_params(seed))
        if case["film"] == "device":
            w, h = case["width"], case["height"]
            state["film"] = {"rgb_sum": torch.empty((h, w, 3), dtype=torch.float32, device="cuda"),
                             "count": torch.empty((h, w), dtype=torch.int32, device="cuda"),
                             "moments": torch.empty((h, w, 2), dtype=torch.float32, device="cuda")}
    elif kind == "batch":
        g = np.random.default_rng(seed)
        state["batch"] = lib.GpuBatch()
        state["integrators"] = []
        for k in range(case["scenes"]):
            s = scenes.cornell_icosphere(freq=int(round(math.exp(g.uniform(math.log(20), math.log(90))))),
                                         width=case["width"], height=case["height"], spp=case["spp"],
                                         max_bounces=case["bounces"], seed=seed + k,
                                         sphere_material=_material(("diffuse", "glass", "gold")[k % 3]))
            s.seed = seed + k
            state["integrators"].append(lib.GpuPathIntegrator(lib.GpuAccel(s, device_sah=True), s))
    else:
        state["guide"] = lib.GpuGuide(GUIDE_AABB, seed=1)
        state["guide"].set_params(_guide_params(seed))
        state["samples"] = _training_batch(case["n"], seed)
    return state


# ------------------------------------------------------------------ one pass

def _hits(out):
    """A closest-hit batch: its records as stored (primitive, t, u, v) and t."""
    return {"records": out.view(torch.int32), "t": out[:, 1]}


def _film(film):
    return {"rgb_sum": film.rgb_sum, "count": film.count, "moments": film.moments}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rays":
        if case["query"] == "any":
            state["accel"].intersect_any_device(state["rays"], state["out"])
            return state["out"]
        state["accel"].intersect_device(state["rays"], state["out"])
        return _hits(state["out"])
    if kind == "host":
        a = state["accel"]
        a.submit_host_ptr(state["closest"].data_ptr(), case["n"], state["hits"].data_ptr())
        a.submit_any_host_ptr(state["any"].data_ptr(), case["n"], state["occluded"].data_ptr())
        a.synchronize()
        return {"closest": _hits(state["hits"]), "any": state["occluded"]}
    if kind == "build":
        method = case["method"]
        a = lib.GpuAccel(state["scene"], device_build=method == "linear", device_sah=method != "linear",
                         split=3.0 if method == "split" else None)
        a.intersect_device(state["rays"], state["out"])
        bounds = a.bounds()
        a.close()
        return {"bounds": bounds, "hits": _hits(state["out"])}
    if kind == "frame":
        integ = state["integrator"]
        strata = case["strata"]
        if case["film"] == "host":
            return _film(integ.render(wave_paths=case["wave"], guide=state.get("guide"),
                                      sampler=abi.BBG_SAMPLER_STRATIFIED if strata else abi.BBG_SAMPLER_INDEPENDENT,
                                      x_samples=strata or 1))
        p, film, out = abi.RenderParams(), abi.Film(), state["film"]
        p.spp, p.seed, p.wave_paths, p.use_graph = case["spp"], integ.scene.seed, case["wave"], 1
        p.sampler = abi.BBG_SAMPLER_STRATIFIED if strata else abi.BBG_SAMPLER_INDEPENDENT
        p.x_samples, p.jitter = strata or 1, 1
        p.guide = state["guide"].h if case["guided"] else None
        film.rgb_sum, film.count, film.moments = (out[k].data_ptr() for k in ("rgb_sum", "count", "moments"))
        integ.render_device(lib.camera(integ.scene.camera), p, film, abi.RenderStats())
        return out
    if kind == "batch":
        films, _ = state["batch"].render(state["integrators"], case["spp"])
        return [_film(f) for f in films]
    grad, loss = state["guide"].gradient(*state["samples"])
    return {"grad": grad, "loss": loss}


# ------------------------------------------------------------------ floors

def _triangles(case):
    return case["size"] if case["scene"] == "soup" else 20 * 4 ** case["size"] + 14


def _trace_flops(triangles, rays):
    """One box of each level of a binary tree (12 operations) and one triangle (50) per ray."""
    return rays * (12.0 * math.log2(max(2, triangles)) + 50.0)


def work(case):
    """Inputs read once and outputs written once; operations of the least
    traversal, one vertex per path, and the network's multiplications."""
    kind = case["kind"]
    if kind == "rays":
        t = _triangles(case)
        return {"bytes": case["n"] * (48 if case["query"] == "closest" else 33) + 36 * t, "flops": _trace_flops(t, case["n"])}
    if kind == "host":
        t = _triangles(case)
        return {"bytes": case["n"] * (48 + 33) + 36 * t, "flops": _trace_flops(t, 2 * case["n"])}
    if kind == "build":
        t = _triangles(case)
        return {"bytes": 36 * t + 64 * t + 48 * case["n"], "flops": 40.0 * t * math.log2(t) + _trace_flops(t, case["n"])}
    if kind in ("frame", "batch"):
        n = case["scenes"] if kind == "batch" else 1
        pixels = n * case["width"] * case["height"]
        paths = pixels * case["spp"]
        t = 100_000 if kind == "batch" else 2 if case["scene"] == "readme" else _triangles(case)
        guide = 2.0 * 15_872 * paths if case.get("guided") else 0.0
        return {"bytes": 24 * pixels + 120 * t * n, "flops": _trace_flops(t, 2 * paths) + 300.0 * paths + guide}
    return {"bytes": 56 * case["n"] + 8 * 16_104, "flops": 6.0 * 15_872 * case["n"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "rays" and case["query"] == "any":
        return "exact"
    if kind in ("rays", "host", "build"):
        # t of the nearest hit to the last bits; which of two primitives hit at
        # exactly the same t is kept may change with the order of the tests.
        return {"rel": 1e-6, "max": 1e-5, "differ": 1e-5}
    if kind == "train":
        # BF16 operands: 32-bit sums in another order round some of them the
        # other way (6.7e-5 and 8e-4 at 16,384 samples, more for fewer).
        return {"rel": 1e-3, "max": 1e-2}
    # A path that meets two primitives at exactly the same t may go on from the
    # other one; everything else repeats to the last bit. Two orders of the same
    # tests (8-wide and binary layout) differ by 9.9e-5 and 0.071 on the
    # 1024 x 1024 frame (189 of 3,145,728 values), by nothing on the others.
    return {"rel": 4e-4, "max": 0.3, "differ": 1e-4}


# ------------------------------------------------------------------ 64 bits

def _exact_hits(scene, rays):
    """t of the nearest triangle hit of every ray (inf: none), in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tri = torch.from_numpy(scene.positions[scene.tri_indices].astype(np.float64)).to(dev)
    p, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    r = torch.from_numpy(rays.astype(np.float64)).to(dev)
    best = torch.empty(r.shape[0], dtype=torch.float64, device=dev)
    step = max(1, (1 << 24) // tri.shape[0])
    for a in range(0, r.shape[0], step):
        o, d = r[a:a + step, None, 0:3], r[a:a + step, None, 3:6]
        lo, hi = r[a:a + step, None, 6], r[a:a + step, None, 7]
        pv = torch.cross(d.expand(-1, tri.shape[0], 3), e2[None].expand(d.shape[0], -1, 3), dim=2)
        inv = 1.0 / (e1[None] * pv).sum(2)
        tv = o - p[None]
        u = (tv * pv).sum(2) * inv
        qv = torch.cross(tv, e1[None].expand_as(tv), dim=2)
        v = (d * qv).sum(2) * inv
        t = (e2[None] * qv).sum(2) * inv
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= lo) & (t <= hi)
        best[a:a + step] = torch.where(ok, t, torch.full_like(t, math.inf)).amin(1)
    return best.cpu()


def _exact_train(params, raw, dirs, weights):
    """Gradient and value of sum_i -w_i log q_i(d_i), the network in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    raw, dirs, weights = (torch.from_numpy(x.astype(np.float64)).to(dev) for x in (raw, dirs, weights))
    parts, at = [], 0
    for s in GUIDE_SHAPES:
        n = int(np.prod(s))
        parts.append(torch.from_numpy(params[at:at + n].astype(np.float64).reshape(s)).to(dev).requires_grad_())
        at += n
    pn = (raw[:, 0:3] + 1.0) * 0.5
    angle = math.pi * pn[:, :, None] * (2.0 ** torch.arange(12, dtype=torch.float64, device=dev))
    x = torch.cat([torch.stack([angle.sin(), angle.cos()], 3).reshape(-1, 72), raw[:, 3:10], torch.ones_like(raw[:, :1])], 1)
    for k in (0, 2, 4):
        x = torch.relu(x @ parts[k].T + parts[k + 1])
    y = (x @ parts[6].T + parts[7]).reshape(-1, 8, 5)
    kappa = y[:, :, 4].clamp(-2.0, 7.0).exp()
    mu = y[:, :, 1:4] / y[:, :, 1:4].norm(dim=2, keepdim=True).clamp_min(1e-6)
    log_norm = kappa.log() - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa))
    log_q = torch.logsumexp(torch.log_softmax(y[:, :, 0], 1) + log_norm +
                            kappa * ((mu * dirs[:, None, :]).sum(2) - 1.0), 1)
    loss = -(weights * log_q).sum()
    loss.backward()
    return torch.cat([p.grad.reshape(-1) for p in parts]).cpu(), float(loss.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind == "rays" and case["query"] == "closest" and _triangles(case) * case["n"] <= 2 ** 28:
        return {"records": None, "t": _exact_hits(_geometry(case, seed), _rays(case, seed + 1)[0])}
    if kind == "train":
        grad, loss = _exact_train(_guide_params(seed), *_training_batch(case["n"], seed))
        return {"grad": grad, "loss": loss}
    return None
