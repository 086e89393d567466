"""The calls whose speed this repository is measured by.

A case is one call that a host application makes: a render of a scene from a
camera, a progressive refinement, the interactive preview, a batch of scenes,
or a query or a training call of the radiance cache. Scenes are seeded and
synthetic, of the same kinds and sizes as hdcodex_b200/workloads.py and the
tests use: a closed box, terrain with spheres under a dome and area lights,
instanced spheres, dispersive and scattering glass with subsurface and
cut-out leaves, and textured layered materials.

listed() holds the calls themselves, draw() further ones of the same ranges;
prepare() makes what the application holds before the call, run() is the call.
"""
import functools
import math

import numpy as np
import torch

from hdcodex_b200 import workloads
from hdcodex_b200.scene import DISK, DOME, LATLONG, RECT, SPHERE, Instancer, Light, Material, Mesh, Scene, Texture
from hdcodex_b200.tracer import PathTracer, RadianceCache, render_batch

# Sizes. Images: a thumbnail to 1080p; samples per call: one (progressive
# display) to 16 (a final-quality increment); triangles: a box to the
# benchmark's million. Wave and grid sizes: 0 keeps the tracer's defaults,
# "tuned" sets what hdcx_autotune picks for a large frame.
MOST_PATHS = 1920 * 1080 * 16 * 3


def _case(name, call, scene, width, height, spp, bounces=8, triangles=0, lights=0, tuned=False, jobs=0, count=0, log2=0,
          steps=0):
    return {"name": name, "call": call, "scene": scene, "width": width, "height": height, "spp": spp, "bounces": bounces,
            "triangles": triangles, "lights": lights, "tuned": tuned, "jobs": jobs, "count": count, "log2": log2,
            "steps": steps}


def listed():
    return [
        # A camera drag in a small viewport: half-resolution, two bounces.
        _case("preview-box-192x128", "preview", "box", 192, 128, 1, bounces=2),
        # The closed 34-triangle box of the benchmark, whole call.
        _case("box-256x256-16spp", "render", "box", 256, 256, 16),
        # The same box lit by an emissive quad: next-event estimation of mesh lights.
        _case("mesh-light-box-301x199-8spp", "render", "lamp", 301, 199, 8),
        # A viewport that refines while nothing moves: eight calls of one sample each.
        _case("progressive-960x540-8x1spp", "progressive", "terrain", 960, 540, 8, triangles=120_000, lights=3),
        # A shot with a dome and several area lights at an odd size.
        _case("lights-639x361-8spp", "render", "terrain", 639, 361, 8, triangles=30_000, lights=6),
        # The million-triangle frame under a dome, on the launch shape the autotuner picks.
        _case("terrain-1m-1920x1080-16spp", "render", "terrain", 1920, 1080, 16, triangles=1_000_000, tuned=True),
        # Dispersive, absorbing and scattering glass, subsurface and cut-outs; hits shaded by material.
        _case("glass-1280x720-8spp", "render", "glass", 1280, 720, 8, triangles=200_000, tuned=True),
        # Layered, textured materials with normal maps, coat and sheen.
        _case("textured-800x450-4spp", "render", "textured", 800, 450, 4, triangles=60_000, lights=2),
        # Instancers: the two-level acceleration structure.
        _case("instanced-960x540-4spp", "render", "instanced", 960, 540, 4, triangles=300_000),
        # A farm node's batch: several small scenes in one call.
        _case("batch-6-jobs", "batch", "terrain", 512, 512, 8, triangles=60_000, lights=4, jobs=6),
        # Radiance-cache predictions for the vertices of a wave, default table.
        _case("cache-query-1000003", "query", "cache", 0, 0, 0, count=1_000_003, log2=19),
        # Online training on the suffix samples of a wave, four steps a call.
        _case("cache-train-65536x4", "train", "cache", 0, 0, 0, count=65_536, log2=15, steps=4),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["render"] * 6 + ["progressive", "preview", "batch", "query", "train"])
    if call == "query":
        return _case("", call, "cache", 0, 0, 0, count=spread(20_000, 2_000_000), log2=rng.randint(17, 19))
    if call == "train":
        return _case("", call, "cache", 0, 0, 0, count=spread(10_000, 80_000), log2=rng.randint(14, 16), steps=rng.randint(1, 4))
    kind = "terrain" if call == "batch" else rng.choice(["box", "lamp", "terrain", "terrain", "glass", "textured", "instanced"])
    small = kind in ("box", "lamp")
    width = spread(100, 1920)
    height = max(64, int(width * rng.uniform(0.5, 0.8)))
    spp = 1 if call == "preview" else spread(1, 16)
    triangles = 0 if small else spread(10_000, 400_000)
    jobs = rng.randint(2, 6) if call == "batch" else 0
    # Two-level and glass frames cost about twice a flattened one per path.
    while width * height * spp * 3 * max(jobs, 1) * (4 if kind in ("glass", "instanced", "textured") else 2) > MOST_PATHS:
        if spp > 1:
            spp = (spp + 1) // 2
        else:
            width, height = width * 3 // 4, height * 3 // 4
    bounces = 2 if call == "preview" else rng.randint(3, 12)
    return _case("", call, kind, width, height, spp, bounces, triangles, rng.randint(0, 7) if not small else 0,
                 call == "render" and rng.random() < 0.4, jobs)


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return workloads._icosphere(level)


def _palette(rng):
    """Lambert, GGX dielectric over diffuse and GGX conductor, as the benchmark's terrain has them."""
    mats = []
    for i in range(12):
        rough = float(rng.uniform(0.05, 0.8))
        m = Material(id=f"/m{i}", base_color=rng.uniform(0.1, 0.9, 3).tolist(), roughness=rough, roughness_v=rough)
        if i % 3 == 0:
            m.specular_weight = 0.0
        elif i % 3 == 2:
            m.metalness = 1.0
        mats.append(m)
    return mats


def _ids(rng, mats, n):
    """A material id per triangle."""
    return np.asarray([m.id for m in mats], dtype=object)[rng.integers(0, len(mats), size=n)].tolist()


def _ground(rng, mats, n, uv=False):
    """A displaced grid of 2 (n - 1)^2 triangles."""
    xs = np.linspace(-12.0, 12.0, n)
    x, z = np.meshgrid(xs, xs)
    pts = np.stack([x.ravel(), np.zeros(n * n), z.ravel()], 1)
    pts[:, 1] = 0.6 * workloads._noise3(pts * 0.35, rng, 4)
    i, j = np.meshgrid(np.arange(n - 1), np.arange(n - 1), indexing="ij")
    a = (i * n + j).ravel()
    tris = np.stack([np.stack([a, a + n, a + 1], 1), np.stack([a + 1, a + n, a + n + 1], 1)], 1).reshape(-1, 3)
    mesh = Mesh(id="/ground", positions=pts.astype(np.float32).ravel(), indices=tris.astype(np.uint32).ravel(),
                material_id=mats[0].id, triangle_material_ids=_ids(rng, mats, len(tris)))
    if uv:
        mesh.texcoords = (pts[tris.ravel()][:, [0, 2]] * 0.5).astype(np.float32).ravel()
    return mesh


def _ball(rng):
    verts, faces = _icosphere(3)
    return verts * (1.0 + 0.18 * workloads._noise3(verts * 2.0, rng, 3))[:, None], faces


def _balls(rng, mats, count, uv=False):
    """Displaced spheres of 1,280 triangles above the ground, flattened."""
    pos, idx = [], []
    for k in range(count):
        v, f = _ball(rng)
        r = rng.uniform(0.25, 0.55)
        pos.append(v * r + np.array([rng.uniform(-10.5, 10.5), 1.2 + r, rng.uniform(-10.5, 10.5)]))
        idx.append(f + k * len(v))
    pos, idx = np.concatenate(pos), np.concatenate(idx).astype(np.uint32)
    mesh = Mesh(id="/balls", positions=pos.astype(np.float32).ravel(), indices=idx.ravel(), material_id=mats[0].id,
                triangle_material_ids=_ids(rng, mats, len(idx)))
    if uv:
        mesh.texcoords = pos[idx.ravel()][:, :2].astype(np.float32).ravel()
        n = pos[idx.ravel()] - pos.reshape(count, -1, 3).mean(1).repeat(idx.size // count, 0)
        mesh.normals = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32).ravel()
    return mesh


def _light_rig(scene, rng, lights, dome=(512, 256)):
    """A lat-long dome and `lights` rect, disk and sphere lights."""
    scene.textures.append(Texture(id="dome#hdr", width=dome[0], height=dome[1],
                                  rgba_float=workloads._dome_texture(*dome, int(rng.integers(1 << 30))).ravel()))
    scene.lights.append(Light(id="/dome", type=DOME, texture="dome#hdr", texture_format=LATLONG))
    for k in range(lights):
        kind = (RECT, DISK, SPHERE)[k % 3]
        size = float(rng.uniform(0.3, 1.2))
        scene.lights.append(Light(
            id=f"/light{k}", type=kind, color=rng.uniform(0.6, 1.0, 3).tolist(), intensity=float(rng.uniform(5, 30)),
            position=[float(rng.uniform(-6, 6)), float(rng.uniform(3, 7)), float(rng.uniform(-6, 6))],
            basis_x=[1.0, 0.0, 0.0], basis_y=[0.0, 0.0, 1.0], basis_z=[0.0, 1.0, 0.0], axis_u=[size, 0.0, 0.0],
            axis_v=[0.0, 0.0, size], width=size, height=size, radius=size * 0.5,
            area=size * size if kind == RECT else math.pi * (size * 0.5) ** 2))


def _terrain_camera(rng, width, height):
    eye = (float(rng.uniform(-4, 4)), float(rng.uniform(6, 8)), float(rng.uniform(14, 17)))
    return workloads.look_at_camera(eye, (0.0, 0.0, -1.0), (0.0, 1.0, 0.0), 45.0, width / height)


def _terrain(rng, triangles, lights, instanced=False):
    s = Scene(revision=1, materials=_palette(rng))
    balls = max(1, int(0.3 * triangles / 1280))
    n = max(8, int(math.sqrt((triangles - 1280 * balls if triangles > 1280 * balls else 128) / 2.0)) + 1)
    s.meshes.append(_ground(rng, s.materials, n))
    if not instanced:
        s.meshes.append(_balls(rng, s.materials, balls))
    else:
        for k in range(min(4, balls)):
            v, f = _ball(rng)
            s.meshes.append(Mesh(id=f"/ball{k}", positions=v.astype(np.float32).ravel(), indices=f.ravel(),
                                 material_id=s.materials[0].id, triangle_material_ids=_ids(rng, s.materials, len(f))))
            moved = []
            for _ in range(max(1, balls // 4)):
                r, th = rng.uniform(0.25, 0.55), rng.uniform(0.0, 2.0 * np.pi)
                c, sn = r * np.cos(th), r * np.sin(th)
                moved.append([[c, 0, -sn, 0], [0, r, 0, 0], [sn, 0, c, 0],
                              [rng.uniform(-10.5, 10.5), 1.2 + r, rng.uniform(-10.5, 10.5), 1]])
            s.instancers.append(Instancer(f"/ball{k}", np.array(moved, dtype=np.float64)))
    _light_rig(s, rng, lights)
    return s


def _textured(rng, triangles, lights):
    """Layered closures with sRGB and linear textures, normal maps, coat and both sheen modes."""
    s = Scene(revision=1)
    for k, (w, h) in enumerate(((512, 512), (256, 300), (128, 128))):
        s.textures.append(Texture(id=f"color{k}", source_path="synthetic", width=w, height=h, srgb=True,
                                  rgba=rng.integers(0, 256, w * h * 4).astype(np.uint8)))
        s.textures.append(Texture(id=f"scalar{k}", source_path="synthetic", width=w, height=h,
                                  rgba=rng.integers(40, 220, w * h * 4).astype(np.uint8)))
    n = rng.normal(size=(256 * 256, 3)) * 0.2 + np.array([0.0, 0.0, 1.0])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    texels = np.concatenate([(n * 0.5 + 0.5) * 255, np.full((len(n), 1), 255.0)], 1)
    s.textures.append(Texture(id="normals", source_path="synthetic", width=256, height=256,
                              rgba=texels.astype(np.uint8).ravel()))
    for k in range(9):
        m = Material(id=f"/t{k}", base_color=rng.uniform(0.2, 0.9, 3).tolist(), roughness=float(rng.uniform(0.1, 0.7)),
                     diffuse_model=k % 4, diffuse_roughness=float(rng.uniform(0.0, 0.8)),
                     base_color_texture=f"color{k % 3}")
        m.roughness_v = m.roughness if k % 2 else float(rng.uniform(0.1, 0.7))
        if k % 3 == 0:
            m.normal_texture, m.roughness_texture = "normals", f"scalar{k % 2}"
        if k % 3 == 1:
            m.coat, m.coat_roughness = 0.8, float(rng.uniform(0.02, 0.3))
            m.coat_roughness_v = m.coat_roughness
        if k % 3 == 2:
            m.sheen, m.sheen_mode = 0.6, (k // 3) % 2
        s.materials.append(m)
    balls = max(1, int(0.5 * triangles / 1280))
    s.meshes += [_ground(rng, s.materials, max(8, int(math.sqrt(triangles / 4.0)) + 1), uv=True),
                 _balls(rng, s.materials, balls, uv=True)]
    _light_rig(s, rng, lights)
    return s


def _workload(case, rng):
    """(scene, camera) of a case."""
    kind, w, h = case["scene"], case["width"], case["height"]
    if kind in ("box", "lamp"):
        wl = workloads.closed_box(w, h, emissive_quad=kind == "lamp")
        for m in wl.scene.materials:
            if m.emission_weight == 0.0:
                m.base_color = rng.uniform(0.05, 0.8, 3).tolist()
        return wl.scene, wl.camera
    if kind == "glass":
        level = 6 if case["triangles"] > 120_000 else 5 if case["triangles"] > 40_000 else 4
        segments = max(16, int(math.sqrt(case["triangles"] / 2.0 * 0.5)))
        wl = workloads.spectral_stress(w, h, seed=int(rng.integers(1 << 30)), sphere_level=level,
                                       torus_segments=(segments, segments), leaf_count=2048, dome_size=(512, 256))
        return wl.scene, wl.camera
    if kind == "textured":
        return _textured(rng, case["triangles"], case["lights"]), _terrain_camera(rng, w, h)
    return _terrain(rng, case["triangles"], case["lights"], kind == "instanced"), _terrain_camera(rng, w, h)


# ---------------------------------------------------------------------------
# State and calls
# ---------------------------------------------------------------------------
def _cache_inputs(case, seed):
    """Parameters, query records and targets of the radiance cache, on the host."""
    rng = np.random.default_rng(seed)
    n = case["count"]
    mlp = np.zeros(17408, np.float32)
    mlp[:16384] = rng.uniform(-0.25, 0.25, 16384)
    mlp[16384:16448] = rng.uniform(-0.25, 0.25, 64)  # the one output in use; the padded rows stay zero
    grid = rng.uniform(-0.5, 0.5, 2 * 16 << case["log2"]).astype(np.float32)
    queries = np.zeros((n, 12), np.float32)
    queries[:, 0:3] = rng.random((n, 3), dtype=np.float32)
    for k in (3, 6):
        v = rng.standard_normal((n, 3), dtype=np.float32)
        queries[:, k:k + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    queries[:, 9:11] = rng.random((n, 2), dtype=np.float32)
    targets = rng.lognormal(0.0, 1.0, n).astype(np.float32)
    return mlp, grid, queries, targets


def prepare(case, seed):
    state = {"case": case}
    if case["scene"] == "cache":
        mlp, grid, queries, targets = _cache_inputs(case, seed)
        cache = RadianceCache(0, log2_table_size=case["log2"])
        cache.set_parameters(mlp, grid)
        state |= {"cache": cache, "queries": torch.from_numpy(queries).cuda(), "targets": torch.from_numpy(targets).cuda(),
                  "out": torch.empty(case["count"], device="cuda")}
        torch.cuda.synchronize()
        return state
    jobs = []
    for k in range(max(case["jobs"], 1)):
        scene, camera = _workload(case, np.random.default_rng([seed, k]))
        tracer = PathTracer(0)
        tracer.set_scene(scene)
        if case["tuned"]:
            tracer.set_tuning(wave_paths=48 << 20, trace_blocks_per_sm=64, shade_blocks_per_sm=16,
                              sort_hits=1 if case["scene"] == "glass" else 0)
        image = torch.empty((case["height"], case["width"], 4), pin_memory=True)
        jobs.append((tracer, camera, image))
    state["jobs"] = jobs
    return state


def run(state):
    case = state["case"]
    call, w, h, spp, bounces = case["call"], case["width"], case["height"], case["spp"], case["bounces"]
    if call == "query":
        state["cache"].query(state["queries"].data_ptr(), case["count"], state["out"].data_ptr())
        return state["out"]
    if call == "train":
        loss = state["cache"].train(state["queries"].data_ptr(), state["targets"].data_ptr(), case["count"], case["steps"])
        mlp, grid = state["cache"].parameters()
        return {"loss": loss, "mlp": mlp, "grid": grid}
    if call == "batch":
        render_batch([(t, camera, w, h, 0, bounces, spp, image.numpy()) for t, camera, image in state["jobs"]], graph=True)
        return [image for _, _, image in state["jobs"]]
    tracer, camera, image = state["jobs"][0]
    if call == "preview":
        return tracer.render_preview(camera, w, h)
    if call == "progressive":
        for sample in range(spp):
            tracer.render(camera, w, h, sample, bounces, 1, out=image.data_ptr())
        return image
    tracer.render(camera, w, h, 0, bounces, spp, out=image.data_ptr())
    return image


def work(case):
    """Bytes: the image or predictions written, the scene or records read once.
    Flops: per path about three rays of a tree descent (eight boxes of six
    planes per level of an 8-wide tree) and two shaded vertices; per query the
    128 taps and the network; per training sample three times that and Adam."""
    if case["call"] in ("query", "train"):
        table = 2 * 16 << case["log2"]
        per = 128 * 4 + 2 * 17408
        if case["call"] == "query":
            return {"bytes": case["count"] * 52 + min(2 * table, case["count"] * 512), "flops": case["count"] * per}
        return {"bytes": case["steps"] * (case["count"] * 52 + 30 * table), "flops": case["steps"] * (3 * case["count"] * per + 12 * table)}
    jobs = max(case["jobs"], 1)
    pixels = case["width"] * case["height"] // (4 if case["call"] == "preview" else 1)
    triangles = case["triangles"] or 34
    images = case["spp"] if case["call"] == "progressive" else 1
    depth = max(1.0, math.log(triangles, 8))
    return {"bytes": jobs * (16 * images * case["width"] * case["height"] + 150 * triangles),
            "flops": jobs * pixels * case["spp"] * 3 * (3 * 2 * depth * 96 + 2 * 600)}


# ---------------------------------------------------------------------------
# Values in 64 bits
# ---------------------------------------------------------------------------
def _taps(queries, log2, level):
    """Table indices (n, 8) and trilinear weights (n, 8) of one level of the
    hash grid (16 levels from 16 to 2048 cells per axis)."""
    n = int(math.floor(16 * math.exp((math.log(2048) - math.log(16)) / 15) ** level))
    # The record is binary32 and so is its scaled position: the cell is part of the question.
    s = np.clip(queries[:, :3], 0.0, 1.0) * np.float32(n)
    c = np.minimum(s.astype(np.int64), n - 1)
    f = (s - c).astype(np.float64)
    side, mask = n + 1, (1 << log2) - 1
    idx = np.empty((len(queries), 8), np.int64)
    wt = np.ones((len(queries), 8))
    for k in range(8):
        p = [c[:, a] + ((k >> a) & 1) for a in range(3)]
        if side ** 3 <= mask + 1:
            idx[:, k] = p[0] + side * (p[1] + side * p[2])
        else:
            idx[:, k] = (p[0] ^ (p[1] * 2654435761 & 0xFFFFFFFF) ^ (p[2] * 805459861 & 0xFFFFFFFF)) & mask
        for a in range(3):
            wt[:, k] *= f[:, a] if (k >> a) & 1 else 1.0 - f[:, a]
    return torch.from_numpy(idx + (level << log2)), torch.from_numpy(wt)


def _forward(taps, rest, layers, table):
    """Activations of every layer; the last is the padded output."""
    x = torch.cat([(table[i] * w[:, :, None]).sum(1) for i, w in taps] + [rest], 1)
    acts = [x]
    for k, m in enumerate(layers):
        x = x @ m.T
        x = x.clamp_min(0.0) if k < 4 else x
        acts.append(x)
    return acts


def _layers(mlp):
    cuts = [0, 4096, 8192, 12288, 16384, 17408]
    return [mlp[a:b].reshape(-1, 64) for a, b in zip(cuts, cuts[1:])]


def exact(case, seed):
    """Images have no value in 64 bits: which light, lobe and triangle a path
    meets is decided by binary32 comparisons, so 64-bit arithmetic follows
    other paths. The cache's predictions and training steps have one."""
    if case["scene"] != "cache":
        return None
    mlp, grid, queries, targets = _cache_inputs(case, seed)
    if case["call"] == "query":
        mlp, table = torch.from_numpy(mlp).double(), torch.from_numpy(grid).double().reshape(-1, 2)
        out = []
        for a in range(0, len(queries), 65536):
            q = queries[a:a + 65536]
            rest = torch.zeros(len(q), 32, dtype=torch.float64)
            rest[:, :9] = torch.from_numpy(q[:, 3:12]).double()
            out.append(_forward([_taps(q, case["log2"], k) for k in range(16)], rest, _layers(mlp), table)[-1][:, 0])
        return torch.cat(out)
    p = [torch.from_numpy(mlp).double(), torch.from_numpy(grid).double()]
    moment, square = [torch.zeros_like(v) for v in p], [torch.zeros_like(v) for v in p]
    y = torch.from_numpy(targets).double()
    taps = [_taps(queries, case["log2"], k) for k in range(16)]
    rest = torch.zeros(len(queries), 32, dtype=torch.float64)
    rest[:, :9] = torch.from_numpy(queries[:, 3:12]).double()
    for step in range(1, case["steps"] + 1):
        layers = _layers(p[0])
        acts = _forward(taps, rest, layers, p[1].reshape(-1, 2))
        pred = acts[-1][:, 0]
        den = pred * pred + 0.01  # held constant in the gradient
        loss = float(((pred - y) ** 2 / den).mean())
        g = torch.zeros_like(acts[-1])
        g[:, 0] = 2.0 * (pred - y) / den / len(y)
        dmlp = [None] * 5
        for k in range(4, -1, -1):
            dmlp[k] = (g.T @ acts[k]).reshape(-1)
            g = g @ layers[k]
            if k:
                g = g * (acts[k] > 0)
        dgrid = torch.zeros(p[1].numel() // 2, 2, dtype=torch.float64)
        for k, (i, w) in enumerate(taps):
            dgrid.index_add_(0, i.reshape(-1), (w[:, :, None] * g[:, None, 2 * k:2 * k + 2]).reshape(-1, 2))
        for k, d in enumerate((torch.cat(dmlp), dgrid.reshape(-1))):  # Adam, the cache's default rates
            moment[k] = 0.9 * moment[k] + 0.1 * d
            square[k] = 0.99 * square[k] + 0.01 * d * d
            p[k] = p[k] - 1e-2 * (moment[k] / (1 - 0.9 ** step)) / ((square[k] / (1 - 0.99 ** step)).sqrt() + 1e-8)
    return {"loss": loss, "mlp": p[0], "grid": p[1]}
