"""Performance cases of the ray queries, the integrators and the path-guiding model.

listed()             the cases, each a dict of plain values
draw(rng)            one more case of the same ranges
prepare(case, seed)  what a caller holds before the call: a scene on the device, rays or a camera, output buffers
run(state)           one pass through the public entry points, and its outputs
work(case)           bytes and operations one pass cannot do without
exact(case, seed)    the outputs in 64-bit arithmetic, where they have such values

The scenes are this package's own workloads (swpathtracer_b200.scenes).  A scene is built once per
process and kept, as a program that renders or queries it again and again does; rays, cameras, sample
seeds and model parameters come from the seed.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import swpathtracer_b200 as spt
from swpathtracer_b200 import abi, scenes

# camera paths per second do not depend on the sample count, so renders use few samples per pixel
LISTED = [
    # A handful of rays against a small scene: picking, collision probes.  Launch latency.
    {"name": "query_257", "kind": "query", "scene": "mesh", "subdiv": 3, "rays": 257},
    # A batch smaller than one full wave of the chip over the 1.31M-triangle mesh: one bounce of a host
    # renderer's tile, a visibility batch.
    {"name": "query_300k", "kind": "query", "scene": "mesh", "subdiv": 8, "rays": 300007},
    # The headline query: 2^24 incoherent rays against 1,310,720 triangles.
    {"name": "query_16m", "kind": "query", "scene": "mesh", "subdiv": 8, "rays": 1 << 24},
    # Rays and hits in page-locked host memory, the reference's 24-byte ray layout, ragged against the
    # pipeline's chunks: a CPU program that offloads its queries.
    {"name": "query_host_3m", "kind": "query_host", "scene": "mesh", "subdiv": 8, "rays": 3000017},
    # The normal ray caster at full HD over the large mesh: an interactive view.
    {"name": "cast_normal_1080p", "kind": "cast", "scene": "mesh", "subdiv": 8, "mode": "normal", "width": 1920,
     "height": 1080},
    # The hit-count caster (the reference's exhaustive traversal), an odd image size.
    {"name": "cast_count_1277x719", "kind": "cast", "scene": "mesh", "subdiv": 8, "mode": "count", "width": 1277,
     "height": 719},
    # A thumbnail of two spheres with a layered material under Russian roulette: the smallest render.
    {"name": "path_plastic_64", "kind": "path", "scene": "furnace_plastic", "subdiv": 0, "width": 64, "height": 64,
     "spp": 4, "end": "russian-roulette", "length": 3, "cap": 0, "sampler": "uniform"},
    # The CPU-runnable path-tracing configuration: the open box with a rough-conductor icosphere.
    {"name": "path_box_256", "kind": "path", "scene": "box", "subdiv": 5, "width": 256, "height": 256, "spp": 16,
     "end": "max-length", "length": 5, "cap": 0, "sampler": "jittered"},
    # The full path-tracing configuration at 1.31M triangles with the coated conductor.
    {"name": "path_layered_800x600", "kind": "path", "scene": "layered", "subdiv": 8, "width": 800, "height": 600,
     "spp": 16, "end": "russian-roulette", "length": 3, "cap": 16, "sampler": "jittered"},
    # Uneven scenes rendered as one batch (every material kind, trees built on the device).
    {"name": "batch_8", "kind": "batch", "scenes": 8, "spp": 4},
    # A render with a frozen guide, as the last pass of a guided render traces most of its samples.
    {"name": "guided_128", "kind": "guided", "scene": "window", "subdiv": 4, "width": 128, "height": 128, "spp": 64,
     "length": 5},
    # The guide's gradients for the configured batch of training records.
    {"name": "guide_gradients_2e18", "kind": "gradients", "records": 1 << 18},
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query_host", "cast", "cast", "path", "path", "path", "batch", "guided",
                       "gradients"])
    if kind in ("query", "query_host"):
        n = _log(rng, 1, 1 << 23) if kind == "query" else _log(rng, 1 << 10, 1 << 22)
        scene = rng.choice(["mesh", "mesh", "smooth"])
        return {"kind": kind, "scene": scene, "subdiv": rng.randint(2, 8) if scene == "mesh" else rng.randint(2, 6),
                "rays": n}
    if kind == "cast":
        scene = rng.choice(["mesh", "mesh", "smooth"])
        return {"kind": kind, "scene": scene, "subdiv": rng.randint(2, 8) if scene == "mesh" else rng.randint(2, 6),
                "mode": rng.choice(["normal", "depth", "count"]), "width": _log(rng, 17, 1920),
                "height": _log(rng, 13, 1080)}
    if kind == "path":
        scene = rng.choice(["box", "layered", "smooth", "furnace_plastic", "furnace_coating", "furnace_lambertian"])
        rr = rng.random() < 0.5
        w, h = _log(rng, 24, 800), _log(rng, 24, 600)
        return {"kind": kind, "scene": scene, "subdiv": 0 if scene.startswith("furnace") else rng.randint(2, 7),
                "width": w, "height": h, "spp": rng.choice([1, 4, 9, 16]),
                "end": "russian-roulette" if rr else "max-length", "length": rng.randint(2, 6),
                "cap": rng.choice([0, 16]) if rr else 0, "sampler": rng.choice(["uniform", "regular", "jittered"])}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 7), "spp": rng.choice([1, 4, 9])}
    if kind == "guided":
        return {"kind": kind, "scene": rng.choice(["window", "small_light"]), "subdiv": rng.randint(2, 5),
                "width": _log(rng, 32, 200), "height": _log(rng, 32, 200), "spp": rng.choice([4, 16, 36]),
                "length": rng.randint(3, 6)}
    return {"kind": "gradients", "records": _log(rng, 77, 1 << 18)}


# ---- scenes ------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _device():
    return spt.Device(0)


def _builder(name, subdiv):
    if name == "mesh":
        return scenes.displaced_mesh_scene(subdiv)
    if name == "smooth":
        return scenes.smooth_mesh_scene(subdiv)
    if name == "box":
        return scenes.box_scene(subdiv)
    if name == "layered":
        return scenes.layered_box_scene(subdiv)
    if name == "window":
        return scenes.window_room_scene(subdivisions=subdiv)
    if name == "small_light":
        return scenes.small_light_box_scene(subdiv)
    return scenes.furnace_scene(name.split("_", 1)[1])


@functools.lru_cache(maxsize=None)
def _packed(name, subdiv):
    return _builder(name, subdiv).build()


@functools.lru_cache(maxsize=None)
def _scene(name, subdiv):
    """The scene on the device, over the reference's own tree (built on the host)."""
    return spt.GpuScene(_device(), _packed(name, subdiv))


@functools.lru_cache(maxsize=None)
def _batch(n):
    """n scenes of the uneven batch, over trees built on the device: [(scene, resolution)]."""
    out = []
    for sb, cam, _, _ in scenes.batched_scenes(n):
        packed = sb.build()
        bvh = spt.Bvh(packed, device=_device())
        out.append((spt.GpuScene(_device(), packed, bvh), cam.width))
        bvh.close()
    return out


def _tris(case):
    if case["scene"].startswith("furnace"):
        return 2
    return 20 * 4 ** case["subdiv"] + (0 if case["scene"] == "mesh" else 12)


# ---- inputs ------------------------------------------------------------------------------------

def _jitter(seed):
    """Three numbers in [-1, 1) that move a camera a little."""
    return np.random.Generator(np.random.Philox(seed)).uniform(-1.0, 1.0, 3)


def _rays(case, seed):
    """Incoherent rays: origins uniform in a cube around the scene, directions uniform on the sphere."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    half, centre = (1.5, 0.0) if case["scene"] == "mesh" else (0.6, 0.5)
    u = torch.rand((n, 5), generator=g, device="cuda", dtype=torch.float32)
    r = torch.zeros((n, 8), device="cuda", dtype=torch.float32)
    r[:, 0:3] = (u[:, 0:3] * 2.0 - 1.0) * half + centre
    z = 1.0 - 2.0 * u[:, 3]
    s = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    r[:, 4] = s * torch.cos(2.0 * math.pi * u[:, 4])
    r[:, 5] = s * torch.sin(2.0 * math.pi * u[:, 4])
    r[:, 6] = z
    return r


def _cast_camera(case, seed):
    j = _jitter(seed)
    if case["scene"] == "mesh":
        return dict(position=(0.35 + 0.1 * j[0], 0.4 + 0.1 * j[1], 3.0 + 0.1 * j[2]), look_at=(0.0, 0.0, 0.0), fov=40.0)
    return dict(position=(0.5 + 0.05 * j[0], 0.5 + 0.05 * j[1], 2.35 + 0.05 * j[2]), look_at=(0.5, 0.5, 0.0), fov=40.0)


def _path_camera(case, seed):
    j = _jitter(seed)
    if case["scene"].startswith("furnace"):
        w = 1.25 + 0.1 * j[0]
        return scenes.camera("orthographic", position=(0, 0, 6), look_at=(0, 0, 0), width=case["width"],
                             height=case["height"], window=(-w, w, -w, w))
    s = 3.0 if case["scene"] == "layered" else 1.0
    return scenes.camera("pinhole", position=((0.5 + 0.05 * j[0]) * s, (0.5 + 0.05 * j[1]) * s, (2.35 + 0.05 * j[2]) * s),
                         look_at=(0.5 * s, 0.5 * s, 0.0), fov=40.0, width=case["width"], height=case["height"])


def _guide_params(seed):
    """Parameters of a guide whose lobes lean around the surface normal (kappa 3 to 10), a little
    different from place to place: the network's hidden layers hand the normal's positive and negative
    parts through, and the last layer tilts one lobe each way.  A trained guide's lobes are about as
    wide; a random network's point below the surface half the time."""
    g = np.random.Generator(np.random.Philox(seed))
    grid = (g.random(abi.GUIDE_GRID_PARAMS, dtype=np.float32) - 0.5) * 0.2
    w = [0.02 * g.standard_normal(s).astype(np.float32) for s in abi.GUIDE_MLP_SHAPES]
    for k in range(3):
        w[0][k, 32 + k] += 1.0       # inputs 32..34: the normal
        w[0][3 + k, 32 + k] -= 1.0
        for h in (1, 2, 3):
            w[h][k, k] += 1.0
            w[h][3 + k, 3 + k] += 1.0
    for lobe in range(8):
        tilt = np.eye(3) + 0.6 * g.uniform(-1.0, 1.0, (3, 3))
        w[4][5 * lobe:5 * lobe + 3, 0:3] += tilt
        w[4][5 * lobe:5 * lobe + 3, 3:6] -= tilt
        w[4][5 * lobe + 3, 0:6] += 1.2
    return grid, np.concatenate([x.ravel() for x in w])


def _records(n, seed):
    """Training records: positions in the unit box, unit directions, sampled directions on the normal's
    side, weights with the long tail that radiance estimates have."""
    g = np.random.Generator(np.random.Philox(seed))
    r = np.zeros(n, abi.GUIDE_RECORD_DTYPE)
    r["pos"] = g.uniform(0.02, 0.98, (n, 3))
    for k in ("normal", "wo", "wi"):
        v = g.standard_normal((n, 3))
        r[k] = v / np.linalg.norm(v, axis=1, keepdims=True)
    for k in ("wo", "wi"):
        r[k] *= np.where((r[k] * r["normal"]).sum(1) < 0.0, -1.0, 1.0)[:, None].astype(np.float32)
    r["weight"] = g.exponential(1.0, n) ** 2
    return r


_MODES = {"normal": abi.RAYCAST_NORMAL, "depth": abi.RAYCAST_DEPTH, "count": abi.RAYCAST_COUNT}


def prepare(case, seed):
    kind = case["kind"]
    dev = _device()
    if kind == "query":
        return {"kind": kind, "scene": _scene(case["scene"], case["subdiv"]), "rays": _rays(case, seed), "n": case["rays"],
                "hits": torch.empty((case["rays"], 4), dtype=torch.int32, device="cuda")}
    if kind == "query_host":
        r = _rays(case, seed)
        rays = torch.cat([r[:, 0:3], r[:, 4:7]], 1).cpu().pin_memory()
        hits = torch.empty((case["rays"], 4), dtype=torch.int32).pin_memory()
        return {"kind": kind, "scene": _scene(case["scene"], case["subdiv"]), "rays": rays.numpy(), "hits": hits,
                "out": hits.numpy().view(abi.HIT_DTYPE).reshape(-1), "keep": rays}
    if kind == "cast":
        w, h = case["width"], case["height"]
        shape, dt = {"normal": ((h, w, 3), torch.float32), "depth": ((h, w), torch.float32),
                     "count": ((h, w), torch.int64)}[case["mode"]]
        return {"kind": kind, "scene": _scene(case["scene"], case["subdiv"]), "mode": _MODES[case["mode"]],
                "cam": scenes.camera("pinhole", width=w, height=h, **_cast_camera(case, seed)),
                "out": torch.empty(shape, dtype=dt, device="cuda")}
    if kind == "path":
        params = scenes.pt_params(spp=case["spp"], sampler=case["sampler"], termination=case["end"],
                                  path_length=case["length"], max_depth=case["cap"], seed=seed)
        return {"kind": kind, "scene": _scene(case["scene"], case["subdiv"]), "cam": _path_camera(case, seed),
                "params": params,
                "image": torch.empty((case["height"], case["width"], 3), dtype=torch.float32, device="cuda")}
    if kind == "batch":
        jobs, images = [], []
        for i, (gs, res) in enumerate(_batch(case["scenes"])):
            jobs.append((gs, scenes.box_camera(res, res),
                         scenes.pt_params(spp=case["spp"], sampler="jittered", termination="max-length", path_length=5,
                                          seed=131 * seed + i)))
            images.append(torch.empty((res, res, 3), dtype=torch.float32, device="cuda"))
        return {"kind": kind, "jobs": jobs, "images": images, "ptrs": [t.data_ptr() for t in images]}
    if kind == "guided":
        guide = spt.Guide(dev, spt.guide_config(max_steps=0, seed=1))
        guide.set_params(*_guide_params(seed))
        return {"kind": kind, "scene": _scene(case["scene"], case["subdiv"]), "cam": _path_camera(case, seed),
                "params": scenes.pt_params(spp=case["spp"], sampler="jittered", termination="max-length",
                                           path_length=case["length"], seed=seed),
                "guide": guide,
                "image": torch.empty((case["height"], case["width"], 3), dtype=torch.float32, device="cuda")}
    n = case["records"]
    guide = spt.Guide(dev, spt.guide_config(batch=n, max_steps=0, seed=1, cache_res=4))
    guide.set_params(*_guide_params(seed))
    return {"kind": kind, "guide": guide, "n": n,
            "recs": torch.from_numpy(_records(n, seed).view(np.uint8).copy()).pin_memory(),
            "grid": torch.empty(abi.GUIDE_GRID_PARAMS, dtype=torch.float32).pin_memory(),
            "mlp": torch.empty(abi.GUIDE_MLP_PARAMS, dtype=torch.float32).pin_memory()}


# ---- one pass ----------------------------------------------------------------------------------

def _hits(h):
    f = h.view(torch.float32)
    return {"t": f[:, 0], "prim": h[:, 1], "uv": f[:, 2:4]}


def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "query":
        state["scene"].intersect_device(state["rays"].data_ptr(), state["n"], state["hits"].data_ptr(), stream)
        return _hits(state["hits"])
    if kind == "query_host":
        state["scene"].intersect(state["rays"], out=state["out"])
        return _hits(state["hits"])
    if kind == "cast":
        state["scene"].raycast_device(state["cam"], state["mode"], state["out"].data_ptr(), stream)
        return state["out"]
    if kind == "path":
        st = state["scene"].pathtrace_device(state["cam"], state["params"], state["image"].data_ptr())
        return {"image": state["image"], "segments": int(st.segments)}
    if kind == "batch":
        st = spt.render_batch(_device(), state["jobs"], state["ptrs"])
        return {"images": state["images"], "segments": int(st[0].segments)}
    if kind == "guided":
        st = state["scene"].pathtrace_guided_device(state["cam"], state["params"], state["guide"],
                                                    state["image"].data_ptr())
        return {"image": state["image"], "segments": int(st.segments)}
    # the C entry point with page-locked buffers (Guide.gradients allocates its result arrays)
    g, loss = state["guide"], ctypes.c_float()
    g.dev.check(g.lib.spt_guide_gradients(g.dev.h, g.h, state["recs"].data_ptr(), state["n"], state["grid"].data_ptr(),
                                          state["mlp"].data_ptr(), ctypes.byref(loss)), "spt_guide_gradients")
    return {"grid": state["grid"], "mlp": state["mlp"], "loss": float(loss.value)}


# ---- what a pass cannot do without -------------------------------------------------------------

def _trace_flops(rays, tris):
    """The boxes of one root-to-leaf descent of an 8-wide tree (8 boxes a level, 12 operations each) and
    one triangle test."""
    return rays * (96.0 * max(1.0, math.log(max(tris, 2), 8)) + 50.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = [(cam.width, sb.arrays()[0].shape[0]) for sb, cam, _, _ in _batch_shapes(case["scenes"])]
        paths = sum(r * r * case["spp"] for r, _ in sizes)
        return {"bytes": sum(12.0 * r * r + 36.0 * t for r, t in sizes),
                "flops": _trace_flops(2.0 * paths, max(t for _, t in sizes))}
    if kind == "gradients":
        n = case["records"]
        return {"bytes": 64.0 * n + 4.0 * (abi.GUIDE_GRID_PARAMS + abi.GUIDE_MLP_PARAMS) * 2.0,
                "flops": 6.0 * abi.GUIDE_MLP_PARAMS * n}
    tris = _tris(case)
    if kind in ("query", "query_host"):
        n, per = case["rays"], 48.0 if kind == "query" else 40.0
        return {"bytes": per * n + 36.0 * tris, "flops": _trace_flops(n, tris)}
    px = case["width"] * case["height"]
    if kind == "cast":
        return {"bytes": {"normal": 12.0, "depth": 4.0, "count": 8.0}[case["mode"]] * px + 36.0 * tris,
                "flops": _trace_flops(px, tris)}
    return {"bytes": 12.0 * px + 36.0 * tris, "flops": _trace_flops(2.0 * px * case["spp"], tris)}


@functools.lru_cache(maxsize=None)
def _batch_shapes(n):
    return scenes.batched_scenes(n)


# ---- 64-bit values -----------------------------------------------------------------------------

def _closest64(packed, o, d):
    """Closest hits of rays (float64, on the GPU) by testing every triangle: t, u, v (t = inf: none)."""
    tri = torch.from_numpy(packed.data).cuda().double().reshape(-1, 3, 3)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = o.shape[0]
    best = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    arg = torch.zeros(n, dtype=torch.int64, device="cuda")
    uv = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 23) // len(v0))
    for a in range(0, n, step):
        ro, rd = o[a:a + step, None, :], d[a:a + step, None, :]
        p = torch.linalg.cross(rd.expand(-1, len(v0), -1), e2[None].expand(rd.shape[0], -1, -1))
        det = (p * e1[None]).sum(-1)
        inv = 1.0 / det
        s = ro - v0[None]
        u = (s * p).sum(-1) * inv
        q = torch.linalg.cross(s, e1[None].expand(rd.shape[0], -1, -1))
        v = (rd * q).sum(-1) * inv
        t = (q * e2[None]).sum(-1) * inv
        ok = (det.abs() >= 1e-6) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 0)
        t = torch.where(ok, t, math.inf)
        best[a:a + step], arg[a:a + step] = t.min(1)
        k = arg[a:a + step, None]
        hit = torch.isfinite(best[a:a + step])
        uv[a:a + step, 0] = torch.where(hit, u.gather(1, k)[:, 0], 0.0)
        uv[a:a + step, 1] = torch.where(hit, v.gather(1, k)[:, 0], 0.0)
    return best, arg, uv


def _unit(v):
    return v / np.linalg.norm(v)


def _gradients64(case, seed):
    n = case["records"]
    grid, mlp = _guide_params(seed)
    rec = _records(n, seed)
    to = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda().double()  # noqa: E731
    grid = to(grid).reshape(abi.GUIDE_LEVELS, abi.GUIDE_T, abi.GUIDE_FEATS).requires_grad_()
    weights, at = [], 0
    for s in abi.GUIDE_MLP_SHAPES:
        weights.append(to(mlp[at:at + s[0] * s[1]].reshape(s)).requires_grad_())
        at += s[0] * s[1]
    total = float(rec["weight"].astype(np.float64).sum()) / n
    loss = 0.0
    growth = math.exp(math.log(1024 / 16) / 15)
    for a in range(0, n, 1 << 16):
        r = rec[a:a + (1 << 16)]
        pos, m = to(r["pos"]).clamp(0.0, 0.99999994), len(r)
        feats = []
        for lv in range(abi.GUIDE_LEVELS):
            res = int(math.floor(16 * growth ** lv + 1e-6))
            x = pos * res
            f = x.floor()
            w, i = x - f, f.long()
            acc = 0.0
            for c in range(8):
                b = [(c >> k) & 1 for k in range(3)]
                g = [i[:, k] + b[k] for k in range(3)]
                if (res + 1) ** 3 <= abi.GUIDE_T:
                    idx = g[0] + g[1] * (res + 1) + g[2] * (res + 1) ** 2
                else:
                    idx = (g[0] ^ (g[1] * 2654435761) ^ (g[2] * 805459861)) & (abi.GUIDE_T - 1)
                cw = 1.0
                for k in range(3):
                    cw = cw * (w[:, k] if b[k] else 1.0 - w[:, k])
                acc = acc + cw[:, None] * grid[lv][idx]
            feats.append(acc)
        h = torch.cat(feats + [to(r["normal"]), to(r["wo"]), torch.zeros((m, 10), dtype=torch.float64, device="cuda")], 1)
        for k, wk in enumerate(weights):
            h = h @ wk.T
            if k < 4:
                h = torch.relu(h)
        y = h[:, :40].reshape(m, 8, 5)
        mu = y[:, :, 0:3] / y[:, :, 0:3].norm(dim=2, keepdim=True).clamp(min=1e-12)
        kappa = torch.exp(y[:, :, 3].clamp(-2.3, 7.0))
        cosine = (mu * to(r["wi"])[:, None, :]).sum(2)
        pdf = kappa / (2.0 * math.pi * (1.0 - torch.exp(-2.0 * kappa))) * torch.exp(kappa * (cosine - 1.0))
        q = (torch.softmax(y[:, :, 4], 1) * pdf).sum(1).clamp(min=1e-30)
        part = (-(to(r["weight"]) / total) * torch.log(q)).sum() / n
        part.backward()
        loss += float(part)
    return {"grid": grid.grad.reshape(-1).cpu(), "mlp": torch.cat([wk.grad.reshape(-1) for wk in weights]).cpu(),
            "loss": loss}


def exact(case, seed):
    """Path-traced images have no 64-bit value: every sample's path hangs on comparisons of its random
    numbers with rounded probabilities.  Hits do, where testing every triangle is quick."""
    kind = case["kind"]
    if kind == "gradients":
        return _gradients64(case, seed)
    if kind not in ("query", "query_host", "cast") or case["scene"] != "mesh":
        return None
    n = case["rays"] if "rays" in case else case["width"] * case["height"]
    if case.get("mode") == "count" or n * _tris(case) > 1 << 31:
        return None
    packed = _packed(case["scene"], case["subdiv"])
    if kind != "cast":
        r = _rays(case, seed).double()
        t, _, uv = _closest64(packed, r[:, 0:3], r[:, 4:7])
        return {"t": t, "prim": None, "uv": uv}
    w, h, c = case["width"], case["height"], _cast_camera(case, seed)
    pos = np.float32(c["position"]).astype(np.float64)
    look, up = np.float32(c["look_at"]).astype(np.float64), np.array([0.0, 1.0, 0.0])
    back = _unit(pos - look)
    right = _unit(np.cross(up, back))
    top = np.cross(back, right)
    far = (0.5 * h) / math.tan(0.5 * c["fov"] * math.pi / 180.0)
    xs = torch.arange(w, dtype=torch.float64, device="cuda") + 0.5 - 0.5 * w
    ys = 0.5 * h - (torch.arange(h, dtype=torch.float64, device="cuda") + 0.5)
    basis = [torch.from_numpy(v).cuda() for v in (right, top, back)]
    d = xs[None, :, None] * basis[0] + ys[:, None, None] * basis[1] - far * basis[2]
    d = (d / d.norm(dim=2, keepdim=True)).reshape(-1, 3)
    t, k, _ = _closest64(packed, torch.from_numpy(pos).cuda().expand(w * h, 3), d)
    hit = torch.isfinite(t)
    if case["mode"] == "depth":
        return torch.where(hit, t, -1.0).reshape(h, w)
    tri = torch.from_numpy(packed.data).cuda().double().reshape(-1, 3, 3)
    nrm = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    return torch.where(hit[:, None], nrm[k], 0.0).reshape(h, w, 3)
