"""Performance cases: what a program that renders with this framework has it do.

Each case is a dict of plain values.  Its "op" names the call sequence:
  render  a resident scene rendered into a film and read back (Stage.render, Film.read)
  scene   a scene that has just been made or changed: Stage(prims), a short render, read back
  rays    a caller's own rays: Stage.intersect and Stage.visibility on host arrays
  batch   several images in one render_batch call, every film read back
  serve   requests submitted to a Server, stepped until done and taken

Scenes are the seeded synthetic scenes of gammaray_gb300.scenes (the Cornell box with two
spheres; the displaced sphere on a ground plane, 1k to 400k triangles), with the seed of
the case in place of the scene's own.  A case's film is cleared before each pass, as a
program does that renders the next frame.
"""
import math

import numpy as np
import torch

import gammaray_gb300 as g
from gammaray_gb300 import batch, scenes, serve

# ------------------------------------------------------------------ cases


def listed():
    return [
        # An interactive preview: one Stage.trace pass of a small image.  Latency and
        # launches are all of it.
        {"name": "preview_pass", "op": "render", "integrator": "pt", "scene": "cornell", "tris": 12, "width": 96,
         "height": 54, "spp": 1, "depth": 8, "attributes": False},
        # The Cornell box configuration: 256 x 256, 16 spp, depth 8.
        {"name": "cornell_256", "op": "render", "integrator": "pt", "scene": "cornell", "tris": 12, "width": 256,
         "height": 256, "spp": 16, "depth": 8, "attributes": False},
        # An ordinary mesh with shading normals and uvs, odd image size, the reference's
        # unbounded depth (roulette ends the paths).
        {"name": "mesh_ragged", "op": "render", "integrator": "pt", "scene": "mesh", "tris": 12_000, "width": 641,
         "height": 359, "spp": 9, "depth": 0, "attributes": True},
        # The headline configuration: 102,400 triangles, 1024 x 1024, 64 spp, depth 12.
        {"name": "mesh_1024", "op": "render", "integrator": "pt", "scene": "mesh", "tris": 102_400, "width": 1024,
         "height": 1024, "spp": 64, "depth": 12, "attributes": False},
        # BDPT with the reference's weights and constants, a small still.
        {"name": "bdpt_reference", "op": "render", "integrator": "bdpt", "scene": "cornell", "tris": 12,
         "width": 200, "height": 150, "spp": 4, "depth": 16, "attributes": False},
        # BDPT with MIS and light tracing: 512 x 512, 16 spp, length 10.
        {"name": "bdpt_mis_512", "op": "render", "integrator": "bdpt_mis", "scene": "mesh", "tris": 102_400,
         "width": 512, "height": 512, "spp": 16, "depth": 10, "attributes": False},
        # A new scene on the reference's host SAH build, then a quick look at it.
        {"name": "scene_host", "op": "scene", "device_build": False, "tris": 102_400, "width": 512, "height": 512,
         "spp": 4},
        # A large, changing scene on the device build.
        {"name": "scene_device", "op": "scene", "device_build": True, "tris": 400_000, "width": 512, "height": 512,
         "spp": 4},
        # Picking: a handful of rays.
        {"name": "rays_small", "op": "rays", "tris": 10_000, "rays": 257},
        # A caller that traces its own rays in bulk.
        {"name": "rays_1m", "op": "rays", "tris": 102_400, "rays": 1 << 20},
        # A batch of images of mixed sizes.
        {"name": "batch_12", "op": "batch", "jobs": 12, "tris": 20_000, "spp": 16, "depth": 8},
        # Requests of mixed sizes on a resident server.
        {"name": "serve_6", "op": "serve", "requests": 6, "tris": 50_000, "spp": 24, "depth": 12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["render", "render", "render", "scene", "rays", "batch", "serve"])
    if op == "render":
        integrator = rng.choice(["pt", "pt", "pt", "bdpt", "bdpt_mis"])
        scene = rng.choice(["cornell", "mesh", "mesh"])
        top = 1024 if integrator == "pt" else 512
        width, height = _log(rng, 33, top), _log(rng, 33, top)
        # samples: up to 64 per pixel for the path tracer and 16 for BDPT
        spp = _log(rng, 1, 64 if integrator == "pt" else 16)
        depth = rng.randint(4, 16) if integrator != "pt" else rng.choice([0, 4, 8, 12])
        if integrator != "pt":  # keep the number of strategies within the largest listed case's
            spp = max(1, min(spp, 16 * 512 * 512 * 100 // (width * height * depth * depth)))
        return {"op": "render", "integrator": integrator, "scene": scene,
                "tris": 12 if scene == "cornell" else _log(rng, 1_000, 200_000), "width": width, "height": height,
                "spp": spp, "depth": depth, "attributes": scene == "mesh" and rng.random() < 0.3}
    if op == "scene":
        dev = rng.random() < 0.5
        return {"op": "scene", "device_build": dev, "tris": _log(rng, 1_000, 400_000 if dev else 100_000),
                "width": _log(rng, 64, 512), "height": _log(rng, 64, 512), "spp": rng.randint(1, 4)}
    if op == "rays":
        return {"op": "rays", "tris": _log(rng, 1_000, 100_000), "rays": _log(rng, 100, 1_000_000)}
    if op == "batch":
        return {"op": "batch", "jobs": rng.randint(3, 12), "tris": _log(rng, 1_000, 20_000), "spp": rng.randint(4, 16),
                "depth": rng.randint(4, 8)}
    return {"op": "serve", "requests": rng.randint(2, 6), "tris": _log(rng, 10_000, 50_000), "spp": rng.randint(4, 24),
            "depth": rng.randint(4, 12)}


# --------------------------------------------------------------- workloads

# Image sizes of the batch and serving mixes, in turn.
BATCH_SIZES = [(128, 128), (256, 256), (512, 512), (333, 217)]
SERVE_SIZES = [(256, 256), (640, 360), (512, 512), (1024, 576)]


def _integrator(kind, depth):
    if kind == "pt":
        return g.PathTracerIntegrator(max_depth=depth)
    if kind == "bdpt":
        return g.BdptIntegrator(max_depth=depth)
    return g.BdptIntegrator(max_depth=depth, mis=1, light_tracing=1)


def _with_attributes(mesh, rings):
    """The displaced sphere with smooth vertex normals and a latitude-longitude uv map."""
    v, t = mesh.vertices, mesh.triangles
    a, b, c = v[t[:, 0]], v[t[:, 1]], v[t[:, 2]]
    n = np.zeros_like(v)
    face = np.cross(a - c, b - c)
    for k in range(3):
        np.add.at(n, t[:, k], face)
    n /= np.maximum(np.linalg.norm(n, axis=1, keepdims=True), 1e-20)
    segments = 2 * rings
    i, j = np.meshgrid(np.arange(rings + 1), np.arange(segments + 1), indexing="ij")
    uv = np.stack([j / segments, i / rings], -1).reshape(-1, 2)
    return g.Mesh(mesh.material, None, v, t, normals=n, tri_normals=t, uvs=uv, tri_uvs=t)


def _workload(scene, tris, width, height, spp, seed, attributes=False):
    if scene == "cornell":
        w = scenes.cornell_spheres(width, height, spp)
        # the seed places the two spheres
        rng = np.random.default_rng(seed)
        for k, s in enumerate(w.prims[2:]):
            s.center = (s.center + rng.uniform(-0.1, 0.1, 3) * (1.0, 0.0, 1.0)).astype(np.float32)
        return w
    w = scenes.displaced_sphere(width, height, spp, seed=seed, tris=tris)
    if attributes:
        rings = max(4, int(round(math.sqrt(tris / 4.0)))) if tris != 102_400 else 160
        w.prims[0] = _with_attributes(w.prims[0], rings)
    return w


# ----------------------------------------------------------------- prepare


def _rays(w, n, seed):
    """Half toward the mesh from a shell around it (as camera and shadow rays come), half
    leaving points near its surface in random directions (as bounces do)."""
    rng = np.random.default_rng(seed)

    def unit(k):
        d = rng.standard_normal((k, 3))
        return d / np.linalg.norm(d, axis=1, keepdims=True)

    k = n // 2
    o1 = unit(k) * 4.0
    d1 = unit(k) * rng.uniform(0.0, 1.1, (k, 1)) - o1
    o2 = unit(n - k) * 1.15
    rays = np.concatenate([np.concatenate([o1, d1 / np.linalg.norm(d1, axis=1, keepdims=True)], 1),
                           np.concatenate([o2, unit(n - k)], 1)]).astype(np.float32)
    pairs = np.concatenate([unit(n) * rng.uniform(1.1, 2.0, (n, 1)), unit(n) * rng.uniform(1.1, 2.0, (n, 1))],
                           1).astype(np.float32)
    return rays, pairs


def prepare(case, seed):
    lib = g.load()
    op = case["op"]
    s = {"op": op, "lib": lib}
    if op == "render":
        w = _workload(case["scene"], case["tris"], case["width"], case["height"], case["spp"], seed,
                      case["attributes"])
        s["stage"] = g.Stage(w.prims, lib=lib, environment=w.environment, seed=seed)
        s["film"] = g.Film(w.width, w.height, lib=lib)
        s["camera"], s["spp"] = w.camera, case["spp"]
        s["integrator"] = _integrator(case["integrator"], case["depth"])
        s["splat"] = case["integrator"] == "bdpt_mis"
    elif op == "scene":
        w = _workload("mesh", case["tris"], case["width"], case["height"], case["spp"], seed)
        s["workload"], s["seed"], s["device_build"] = w, seed, case["device_build"]
        s["film"] = g.Film(w.width, w.height, lib=lib)
    elif op == "rays":
        w = _workload("mesh", case["tris"], 64, 64, 1, seed)
        s["stage"] = g.Stage(w.prims, lib=lib, environment=w.environment, seed=seed)
        s["rays"], s["pairs"] = _rays(w, case["rays"], seed)
    elif op == "batch":
        s["jobs"] = []
        for k in range(case["jobs"]):
            width, height = BATCH_SIZES[k % len(BATCH_SIZES)]
            w = _workload("mesh", case["tris"] // (1 + k % 3), width, height, case["spp"], seed * 64 + k)
            st = g.Stage(w.prims, lib=lib, environment=w.environment, seed=seed + k)
            s["jobs"].append(batch.Job(st, w.camera, g.PathTracerIntegrator(max_depth=case["depth"]),
                                       g.Film(width, height, lib=lib), case["spp"]))
    else:
        s["server"] = serve.Server(lib, path_capacity=1 << 24)
        s["requests"] = []
        for k in range(case["requests"]):
            width, height = SERVE_SIZES[k % len(SERVE_SIZES)]
            w = _workload("mesh", case["tris"] // (1 + k % 3), width, height, case["spp"], seed * 64 + k)
            st = g.Stage(w.prims, lib=lib, environment=w.environment, seed=seed + k)
            s["requests"].append((st, w.camera, g.PathTracerIntegrator(max_depth=case["depth"]), width, height,
                                  case["spp"]))
    return s


# --------------------------------------------------------------------- run


def _film(film):
    accum, weight = film.read()
    return {"accum": accum, "weight": weight}


def run(s):
    op = s["op"]
    if op == "render":
        s["film"].clear()
        if s["spp"] == 1:
            s["stage"].trace(s["camera"], s["integrator"], s["film"])
        else:
            s["stage"].render(s["camera"], s["integrator"], s["film"], s["spp"])
        if s["splat"]:  # the resolved image holds the light-tracing splats
            return {"rgb": s["film"].resolve(), "weight": s["film"].read()[1]}
        return _film(s["film"])
    if op == "scene":
        w = s["workload"]
        s["film"].clear()
        stage = g.Stage(w.prims, lib=s["lib"], environment=w.environment, seed=s["seed"],
                        device_build=s["device_build"])
        stage.render(w.camera, g.PathTracerIntegrator(max_depth=12), s["film"], w.spp)
        out = _film(s["film"])
        stage.close()
        return out
    if op == "rays":
        hits = s["stage"].intersect(s["rays"])
        visible = s["stage"].visibility(s["pairs"])
        return {"t": hits["t"], "prim": hits["prim"], "component": hits["component"], "u": hits["u"],
                "v": hits["v"], "visible": visible}
    if op == "batch":
        for j in s["jobs"]:
            j.film.clear()
        batch.render_batch(s["jobs"], s["lib"])
        return [_film(j.film) for j in s["jobs"]]
    srv = s["server"]
    ids = [srv.submit(*r) for r in s["requests"]]
    srv.run_until_done(ids)
    out = []
    for i in ids:
        accum, weight = srv.take(i)
        out.append({"accum": accum, "weight": weight})
    return out


# -------------------------------------------------------------------- work


def _scene_bytes(tris):
    """A component's 48-byte record and its share of the box tree (about a quarter of a
    128-byte node): what a traversal has to be able to reach."""
    return (tris + 22) * (48 + 32)


# Per traced segment, estimated from traversal counts of the displaced sphere: about 9
# nodes of 4 boxes (6 subtractions, 6 products, 11 comparisons each), 3 triangle tests
# (about 50 operations) and one Disney sample, value and density (about 400).
SEGMENT_FLOPS = 9 * 4 * 23 + 3 * 50 + 400


def work(case):
    op = case["op"]
    if op in ("render", "scene"):
        samples = case["width"] * case["height"] * case["spp"]
        film = 16 * case["width"] * case["height"]
        scene = _scene_bytes(case["tris"])
        if op == "scene":
            scene += 48 * case["tris"]  # vertices and indices in, records out
        segments = 1.7 * samples if case.get("scene") != "cornell" else 4.0 * samples
        if str(case.get("integrator")).startswith("bdpt"):
            segments *= 3.0  # both walks and the connections between them
        # 25 filter taps of 8 operations a sample
        return {"bytes": scene + film, "flops": segments * SEGMENT_FLOPS + samples * 200}
    if op == "rays":
        n = case["rays"]
        return {"bytes": n * (24 + 20 + 24 + 1) + _scene_bytes(case["tris"]), "flops": 2 * n * (SEGMENT_FLOPS - 400)}
    count, sizes = (case["jobs"], BATCH_SIZES) if op == "batch" else (case["requests"], SERVE_SIZES)
    nbytes = flops = 0
    for k in range(count):
        px = sizes[k % len(sizes)][0] * sizes[k % len(sizes)][1]
        nbytes += 16 * px + _scene_bytes(case["tris"] // (1 + k % 3))
        flops += px * case["spp"] * (1.7 * SEGMENT_FLOPS + 200)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------- exact
# In 64 bits there are values for a film's filter weights (they depend on the sample
# positions alone) and for closest hits.  A path's radiance has none: a rounding that
# turns one lobe choice or roulette draw gives another path.


def _mix64(z):
    def shr(x, k):  # logical right shift of int64 bits
        return (x >> k) & ((1 << (64 - k)) - 1)

    def signed(c):
        return c - (1 << 64) if c >= 1 << 63 else c

    z = z + signed(0x9E3779B97F4A7C15)
    z = (z ^ shr(z, 30)) * signed(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * signed(0x94D049BB133111EB)
    return z ^ shr(z, 31)


def _film_weight(width, height, passes, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pixel = torch.arange(width * height, dtype=torch.int64, device=dev)
    row, col = pixel // width, pixel % width
    out = torch.zeros(width * height, dtype=torch.float64, device=dev)

    def uniform(key, dim):
        step = dim * 0xD1B54A32D192ED03 % (1 << 64)
        h = _mix64(key + (step - (1 << 64) if step >= 1 << 63 else step))
        return ((h >> 40) & 0xFFFFFF).double() / 16777216.0

    def mitchell(x):
        x = x.abs()
        b = c = 1.0 / 3.0
        inner = (12 - 9 * b - 6 * c) * x ** 3 + (-18 + 12 * b + 6 * c) * x ** 2 + (6 - 2 * b)
        outer = (-b - 6 * c) * x ** 3 + (6 * b + 30 * c) * x ** 2 + (-12 * b - 48 * c) * x + (8 * b + 24 * c)
        return torch.where(x > 1, outer, inner) / 6.0

    for p in passes:
        key = _mix64(seed ^ _mix64((p << 32) | pixel))
        y = row - 2 + 4 * uniform(key, 0)
        x = col - 2 + 4 * uniform(key, 1)
        x0, x1 = torch.ceil(x - 2).clamp(0, width - 1).long(), torch.floor(x + 2).clamp(0, width - 1).long()
        y0, y1 = torch.ceil(y - 2).clamp(0, height - 1).long(), torch.floor(y + 2).clamp(0, height - 1).long()
        for dy in range(5):
            py = y0 + dy
            wy = torch.where(py <= y1, mitchell(py - y), 0.0)
            for dx in range(5):
                px = x0 + dx
                wx = torch.where(px <= x1, mitchell(px - x), 0.0)
                out.index_add_(0, (py.clamp(max=height - 1) * width + px.clamp(max=width - 1)), wx * wy)
    return out.view(height, width).cpu().numpy()


def _closest_hits(prims, rays):
    """Moller and Trumbore's test of every ray against every triangle: the first positive
    distance (above the renderer's FLT_EPSILON), with the renderer's cut-off for
    near-parallel triangles."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    eps = float(np.finfo(np.float32).eps)
    corner = [np.concatenate([p.vertices[p.triangles[:, k]] for p in prims]) for k in range(3)]
    a, b, c = (torch.from_numpy(x.astype(np.float64)).to(dev) for x in corner)
    e1, e2 = a - c, b - c
    normal = torch.linalg.cross(e1, e2)
    # With m = o x d: det = -d . n, u det = e2 . m + d . (c x e2), v det = -(e1 . m) - d . (c x e1)
    # and t det = (o - c) . n: products of small matrices.
    mu = torch.cat([e2, torch.linalg.cross(c, e2)], 1).T.contiguous()
    mv = -torch.cat([e1, torch.linalg.cross(c, e1)], 1).T.contiguous()
    cn = (c * normal).sum(1)
    r = torch.from_numpy(rays.astype(np.float64)).to(dev)
    n = len(r)
    t_out = torch.zeros(n, dtype=torch.float64, device=dev)
    uv_out = torch.zeros(2, n, dtype=torch.float64, device=dev)
    step = max(1, (1 << 28) // len(a))
    for k in range(0, n, step):
        o, d = r[k:k + step, :3], r[k:k + step, 3:]
        md = torch.cat([torch.linalg.cross(o, d), d], 1)
        det = -(d @ normal.T)
        inv = 1.0 / det
        u, v = (md @ mu).mul_(inv), (md @ mv).mul_(inv)
        t = (o @ normal.T).sub_(cn).mul_(inv)
        miss = (det.abs_() < eps) | (u < 0) | (v < 0) | (u + v > 1) | (t <= eps)
        t.masked_fill_(miss, math.inf)
        best, at = t.min(1)
        hit = best < math.inf
        at = at.unsqueeze(1)
        t_out[k:k + step] = torch.where(hit, best, 0.0)
        uv_out[0, k:k + step] = torch.where(hit, u.gather(1, at).squeeze(1), 0.0)
        uv_out[1, k:k + step] = torch.where(hit, v.gather(1, at).squeeze(1), 0.0)
    return t_out.cpu().numpy(), uv_out.cpu().numpy()


def exact(case, seed):
    op = case["op"]
    if op in ("render", "scene"):
        weight = _film_weight(case["width"], case["height"], range(case["spp"]), seed)
        if case.get("integrator") == "bdpt_mis":
            return {"rgb": None, "weight": weight}
        return {"accum": None, "weight": weight}
    if op == "rays":
        w = _workload("mesh", case["tris"], 64, 64, 1, seed)
        t, uv = _closest_hits(w.prims, _rays(w, case["rays"], seed)[0])
        return {"t": t, "prim": None, "component": None, "u": uv[0], "v": uv[1], "visible": None}
    count, sizes = (case["jobs"], BATCH_SIZES) if op == "batch" else (case["requests"], SERVE_SIZES)
    out = []
    for k in range(count):
        width, height = sizes[k % len(sizes)]
        out.append({"accum": None, "weight": _film_weight(width, height, range(case["spp"]), seed + k)})
    return out
