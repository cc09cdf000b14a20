"""Performance cases: the calls that a program using colvillea_b200 makes, from one small preview frame to a full-HD
batch over 4.7 million triangles, with the neural parts, the ray queries and the scene builds and edits beside them.

listed() names the cases that are timed by default; draw(rng) gives further ones of the same ranges.  A case is a dict
of plain values, prepare(case, seed) builds what a program holds before the call, run(state) is one pass through the
public API, work(case) states the bytes and operations that a pass cannot do without, and exact(case, seed) gives the
64-bit values where an output has one (network outputs and gradients, hit distances in small scenes).
"""
import math

import numpy as np
import torch

import colvillea_b200 as cb
from colvillea_b200 import scenes


def _case(name, kind, **kw):
    return {"name": name, "kind": kind, **kw}


def listed():
    return [
        # A viewer's smallest call: one progressive frame of a small scene at preview size.  Launches and waits count.
        _case("preview_256", "render", scene="spheres", width=256, height=256, spp=1, depth=5, estimator="reference",
              sampler="cdf", integrator="path", two_level=False, restart=False),
        # The reference's own granularity at full HD: one sample per pixel and call, then the film to the host.
        _case("progressive_1080p", "render", scene="terrain", terrain=512, objects=128, dome=1024, width=1920,
              height=1080, spp=1, depth=8, estimator="reference", sampler="alias", integrator="path", two_level=False,
              restart=False),
        # A batch of samples in one call over the largest flattened scene (4.7 M triangles), the throughput workload.
        _case("batch_1080p", "render", scene="terrain", terrain=1024, objects=512, dome=2048, width=1920, height=1080,
              spp=8, depth=8, estimator="reference", sampler="alias", integrator="path", two_level=False, restart=True),
        # The direct-lighting integrator on image textures and normal maps, at an odd film size.
        _case("direct_textured", "render", scene="textured", width=1001, height=563, spp=4, depth=1,
              estimator="reference", sampler="cdf", integrator="direct", two_level=False, restart=True),
        # Long paths (depth 16) over rotated and scaled instances kept as a two-level scene, corrected estimator.
        _case("instances_720p", "render", scene="instances", terrain=384, objects=48, copies=12, dome=1024, width=1280,
              height=720, spp=2, depth=16, estimator="corrected", sampler="alias", integrator="path", two_level=True,
              restart=True),
        # Guided path tracing with a given network: encoding, inference and mixture sampling at every vertex.
        _case("guided_1080p", "guided", scene="spheres", width=1920, height=1080, spp=2, depth=5, mask=7),
        # The radiance cache trained while rendering: records, a training step per sample, cache queries.
        _case("cached_540p", "cached", scene="caustics", dome=1024, width=960, height=540, spp=4, depth=16),
        # Ray queries by a program that brings its own rays (picking, visibility, baking).
        _case("ray_queries", "rays", scene="terrain", terrain=512, objects=128, dome=256, rays=1000003),
        # Inference of the guiding network on a program's own points.
        _case("network_forward", "forward", log2_table=19, rows=100003),
        # One gradient of the guiding network over a program's own records.
        _case("network_gradient", "gradient", log2_table=16, rows=200003),
        # Opening a scene: meshes, textures and emitters in host memory to the first frame.
        _case("open_scene", "open", scene="terrain", terrain=512, objects=128, dome=1024, width=640, height=360, depth=8,
              two_level=False),
        # An animated mesh: new vertices, the tree refitted, one frame.
        _case("edit_scene", "edit", scene="terrain", terrain=512, objects=32, dome=256, width=640, height=360, depth=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 5 + ["guided", "cached", "rays", "forward", "gradient", "open", "edit"])
    if kind == "forward":
        return {"kind": kind, "log2_table": rng.randint(14, 19), "rows": _log(rng, 1, 200000)}
    if kind == "gradient":
        return {"kind": kind, "log2_table": rng.randint(13, 17), "rows": _log(rng, 100, 250000)}
    width = _log(rng, 33, 1920)
    c = {"kind": kind, "width": width, "height": max(17, min(1080, int(width * rng.uniform(0.4, 1.2))))}
    if kind == "guided":
        return {**c, "scene": "spheres", "spp": rng.randint(1, 2), "depth": rng.randint(2, 8), "mask": rng.choice([4, 5, 7])}
    if kind == "cached":
        c["width"], c["height"] = min(960, c["width"]), min(540, c["height"])
        return {**c, "scene": "caustics", "dome": rng.choice([256, 512, 1024]), "spp": rng.randint(1, 4),
                "depth": rng.randint(4, 16)}
    terrain = {"scene": "terrain", "terrain": _log(rng, 64, 512), "objects": _log(rng, 4, 128),
               "dome": rng.choice([256, 512, 1024])}
    if kind == "rays":
        c = {"kind": kind, "rays": _log(rng, 100, 1000000)}
        return {**c, **(terrain if rng.random() < 0.6 else {"scene": "spheres"})}
    c["depth"] = rng.randint(2, 12)
    if kind in ("open", "edit"):
        c["width"], c["height"] = min(800, c["width"]), min(600, c["height"])
        return {**c, **terrain, **({"two_level": rng.random() < 0.3} if kind == "open" else {})}
    scene = rng.choice(["spheres", "terrain", "textured", "instances"])
    if scene == "terrain":
        c.update(terrain)
    elif scene == "instances":
        c.update(scene=scene, terrain=_log(rng, 64, 384), objects=rng.randint(4, 48), copies=rng.randint(2, 12),
                 dome=rng.choice([256, 1024]))
    else:
        c["scene"] = scene
    integrator = rng.choice(["path", "path", "direct"])
    return {**c, "spp": _log(rng, 1, 8), "estimator": rng.choice(["reference", "corrected"]),
            "sampler": rng.choice(["cdf", "alias"]), "integrator": integrator,
            "two_level": scene == "instances" and rng.random() < 0.5, "restart": rng.random() < 0.5}


# --- scenes ---------------------------------------------------------------------------------------------------------
def _instances(seed, width, height, terrain, objects, copies, dome):
    """A terrain and `objects` meshes, each placed `copies` times under random rotations and scales."""
    rng = np.random.default_rng(seed)
    meshes = [scenes.terrain_mesh(terrain, 60.0, 2.5, 5, seed + 202, y0=-1.0)]
    mats = [scenes.Material(scenes.MAT_DIFFUSE, reflectance=(0.45, 0.42, 0.38))]
    inst = [(0, 0, scenes.IDENTITY)]
    for u in range(objects):
        meshes.append(scenes.sphere_mesh(4, (0, 0, 0), 0.6) if u % 2 == 0
                      else scenes.torus_mesh(44, 44, (0, 0, 0), 0.6, 0.2))
        kind = int(rng.integers(0, 3))
        rough = float(math.sqrt(rng.uniform(0.05, 0.4)))
        mats.append([scenes.Material(scenes.MAT_DIFFUSE, reflectance=tuple(float(x) for x in rng.uniform(0.2, 0.8, 3))),
                     scenes.Material(scenes.MAT_METAL, reflectance=(1.0, 1.0, 1.0), roughness=rough,
                                     eta=scenes.GOLD_ETA, k=scenes.GOLD_K),
                     scenes.Material(scenes.MAT_GLASS, roughness=rough, interior_ior=1.5)][kind])
        for _ in range(copies):
            q, _r = np.linalg.qr(rng.normal(size=(3, 3)))
            m = np.concatenate([q * rng.uniform(0.5, 2.0),
                                [[rng.uniform(-50, 50)], [rng.uniform(0.5, 4.0)], [rng.uniform(-30, 60)]]], 1)
            inst.append((len(meshes) - 1, len(mats) - 1, tuple(float(x) for x in m.reshape(-1))))
    lobes = [(d, 2.0, 200.0) for d in scenes.random_upper_dirs(rng, 4)]
    sky = scenes.Emitter(scenes.EMIT_DOME, texels=scenes.hdri(dome, dome // 2, lobes, rng))
    cam = scenes.look_at_camera((0, 3, -10), (0, 0, 0), (0, 1, 0), 45.0, width, height)
    return scenes.Scene(width, height, meshes, inst, mats, [scenes.directional(), sky], cam, max_depth=16, rr_start=3)


def _caustics(seed, width, height, dome):
    """Spheres, most of them rough glass, under one very bright small sun."""
    rng = np.random.default_rng(seed + 7)
    lobe = [(scenes.random_upper_dirs(rng, 1)[0], 0.5, 5000.0)]
    sky = scenes.Emitter(scenes.EMIT_DOME, texels=scenes.hdri(dome, dome // 2, lobe, rng))
    return scenes.config1(seed, width, height, glass_frac=0.6, glass_alpha=(0.01, 0.1), dome=sky)


def _scene(c, seed):
    w, h = c.get("width", 64), c.get("height", 64)
    if c["scene"] == "spheres":
        s = scenes.config1(seed, w, h)
    elif c["scene"] == "textured":
        s = scenes.textured(seed, w, h)
    elif c["scene"] == "caustics":
        s = _caustics(seed, w, h, c["dome"])
    elif c["scene"] == "instances":
        s = _instances(seed, w, h, c["terrain"], c["objects"], c["copies"], c["dome"])
    else:
        s = scenes.config2(seed, w, h, c["terrain"], c["objects"], (c["dome"], c["dome"] // 2))
    if "depth" in c:
        s.max_depth = c["depth"]
    return s


def _film(c):
    return torch.empty((c["height"], c["width"], 4), dtype=torch.float32, pin_memory=True).numpy()


def _open(s, c):
    flags = cb.COMPAT_ALL if c.get("estimator", "reference") == "reference" else 0
    if c.get("sampler") == "alias":
        flags |= cb.DOME_ALIAS
    if c.get("two_level"):
        flags |= cb.TWO_LEVEL
    kind = cb.IntegratorType.WavefrontDirectLighting if c.get("integrator") == "direct" \
        else cb.IntegratorType.WavefrontPathTracing
    return cb.load_scene(s, kind, flags=flags)


# --- network inputs -------------------------------------------------------------------------------------------------
def _unit(rng, n):
    v = rng.standard_normal((n, 3), dtype=np.float32)
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _points(rng, n):
    """(n, 9): positions in the unit box (half of them on a ground plane), normals, outgoing directions."""
    p = rng.random((n, 3), dtype=np.float32)
    p[: n // 2, 1] = 0.25 + 0.02 * p[: n // 2, 1]
    return np.ascontiguousarray(np.concatenate([p, _unit(rng, n), _unit(rng, n)], 1), np.float32)


def _params(rng, log2_table):
    """A network's parameters: hash features and Glorot-uniform weights, as after some training."""
    hash_n = 16 * 2 * (1 << log2_table)
    out = [rng.standard_normal(hash_n, dtype=np.float32) * np.float32(0.1)]
    for i, o in ((96, 64), (64, 64), (64, 64), (64, 64), (64, 48)):
        out.append((rng.random(i * o, dtype=np.float32) * 2 - 1) * np.float32(math.sqrt(6.0 / (i + o))))
    return np.concatenate(out)


def _records(rng, n):
    """(n, 14): points, sampled directions, weights and BSDF pdfs of a path tracer's records."""
    w = np.exp(rng.standard_normal((n, 1), dtype=np.float32))
    pdf = np.float32(0.05) + rng.random((n, 1), dtype=np.float32)
    return np.ascontiguousarray(np.concatenate([_points(rng, n), _unit(rng, n), w, pdf], 1), np.float32)


def _network(c, seed):
    rng = np.random.default_rng(seed)
    params = _params(rng, c["log2_table"])
    if c["kind"] == "forward":
        return params, _points(rng, c["rows"])
    return params, _records(rng, c["rows"])


def _rays(c, seed):
    """(n, 8) rays {origin, tmin, direction, tmax}: half from the camera's place, half between points of the scene."""
    rng = np.random.default_rng(seed + 5)
    n, ext = c["rays"], (4.0 if c["scene"] == "spheres" else 30.0)
    o = rng.uniform([-ext, 0.1, -ext], [ext, 3.0, ext], (n, 3))
    o[: n // 2] = (0.0, 3.0, -10.0)
    t = rng.uniform([-ext, -1.0, -ext], [ext, 2.0, ext], (n, 3))
    d = t - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.empty((n, 8), np.float32)
    rays[:, :3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, 1e-3, d, 100.0
    return rays


# --- the cases ------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("forward", "gradient"):
        params, data = _network(c, seed)
        g = cb.Guide.create(cb.GuideConfig(log2_table=c["log2_table"]))
        g.set_params(params)
        return {"kind": kind, "net": g, "data": data}
    s = _scene(c, seed)
    if kind == "open":
        return {"kind": kind, "scene": s, "case": c, "film": _film(c)}
    if kind == "rays":
        return {"kind": kind, "it": _open(s, c), "rays": _rays(c, seed)}
    if kind == "edit":
        it = _open(s, c)
        m, shapes = s.meshes[0], []
        for k in range(2):
            p = m.positions.copy()
            p[:, 1] += np.float32(0.2) * np.sin(np.float32(0.3 + 0.2 * k) * p[:, 0] + np.float32(seed % 97))
            shapes.append(np.ascontiguousarray(p))
        it.render(1)
        return {"kind": kind, "it": it, "film": _film(c), "shapes": shapes, "at": 0}
    if kind == "guided":
        it = _open(s, {**c, "estimator": "corrected", "sampler": "alias"})
        it.setGuiding(cb.GuideConfig(train_spp=0, class_mask=c["mask"]))
        it.guide().set_params(_params(np.random.default_rng(seed + 3), 19))
    elif kind == "cached":
        it = _open(s, {**c, "estimator": "corrected", "sampler": "alias"})
        it.setRadianceCache(cb.RadianceCacheConfig(train_spp=0, network={"batch": 1 << 19, "learning_rate": 1e-3}))
    else:
        it = _open(s, c)
    return {"kind": kind, "it": it, "film": _film(c), "spp": c["spp"], "restart": c.get("restart", True)}


def run(state):
    kind = state["kind"]
    if kind == "forward":
        return state["net"].forward(state["data"])
    if kind == "gradient":
        loss, grad = state["net"].gradient(state["data"])
        return {"loss": loss, "grad": grad}
    if kind == "rays":
        t, prim, b1, b2 = state["it"].traceRays(state["rays"])
        return {"t": t, "prim": prim, "b1": b1, "b2": b2, "occluded": state["it"].occludedRays(state["rays"])}
    if kind == "open":
        with _open(state["scene"], state["case"]) as it:
            it.render(1)
            return it.readbackFramebuffer(state["film"])
    it = state["it"]
    if kind == "edit":
        state["at"] ^= 1
        it.updateVertices(0, state["shapes"][state["at"]])
        it.render(1)
        return it.readbackFramebuffer(state["film"])
    if state["restart"]:
        it.resetIterationIndex()
    it.render(state["spp"])
    return it.readbackFramebuffer(state["film"])


# --- what a pass cannot do without ----------------------------------------------------------------------------------
# Per traced ray: about 20 eight-wide node tests (6 planes, a multiply and an add each) and 5 triangle tests.
_FLOPS_PER_RAY = 20 * 8 * 14 + 5 * 50
_FLOPS_PER_VERTEX = 400  # shading: BSDF and emitter sampling and evaluation


def _triangles(c):
    if c["scene"] in ("spheres", "textured", "caustics"):
        return 10242
    per = 5060 if c["scene"] == "terrain" else 4496
    return 2 * (c["terrain"] - 1) ** 2 + per * c["objects"]


def _scene_bytes(c):
    tris = _triangles(c)
    dome = c.get("dome", 256)
    return tris * (36 + 24 + 16) + dome * (dome // 2) * 16  # positions, vertex attributes, indices; the dome's texels


def work(case):
    c, kind = case, case["kind"]
    if kind == "forward":
        return {"bytes": c["rows"] * (36 + 192), "flops": 2 * c["rows"] * (96 * 64 + 3 * 64 * 64 + 64 * 48)}
    if kind == "gradient":
        n = 32 * (1 << c["log2_table"]) + 21504
        return {"bytes": c["rows"] * 56 + 8 * n, "flops": 6 * c["rows"] * (96 * 64 + 3 * 64 * 64 + 64 * 48)}
    if kind == "rays":
        return {"bytes": c["rays"] * (64 + 17) + _scene_bytes(c), "flops": 2 * c["rays"] * _FLOPS_PER_RAY}
    paths = c["width"] * c["height"] * c.get("spp", 1)
    direct = c.get("integrator") == "direct"
    closest, shadow = (1.0, 1.2) if direct else (2.2, 1.0)  # rays per path
    flops = paths * ((closest + shadow) * _FLOPS_PER_RAY + closest * _FLOPS_PER_VERTEX)
    nbytes = _scene_bytes(c) + c["width"] * c["height"] * 16
    if kind == "guided":
        flops += paths * 2 * (96 * 64 + 3 * 64 * 64 + 64 * 48)
    if kind == "cached":
        # A query for most paths; per training step 16.8 M parameters with their moments and gradient.
        flops += paths * 2 * (96 * 64 + 64 * 64 + 64 * 16)
        nbytes += c["spp"] * 36 * (1 << 24)
    return {"bytes": nbytes, "flops": flops}


# --- 64-bit values --------------------------------------------------------------------------------------------------
_RES = [math.floor(16.0 * 64.0 ** (l / 15.0) + (0.0 if l < 15 else -1e-9)) for l in range(16)]


def _exact_encode(params, x9, log2_table):
    """(n, 96) 64-bit inputs of the network; the hash features are differentiable in params."""
    T, dev = 1 << log2_table, params.device
    p = x9[:, :3].clamp(0.0, 1.0)
    feats = []
    for l, res in enumerate(_RES):
        x = p * res
        i = torch.minimum(x.floor(), torch.tensor(float(res - 1), dtype=x.dtype, device=dev))
        w, i = x - i, i.long()
        f = 0.0
        for k in range(8):
            q = [i[:, a] + ((k >> a) & 1) for a in range(3)]
            if (res + 1) ** 3 <= T:
                h = q[0] + (res + 1) * (q[1] + (res + 1) * q[2])
            else:
                h = (q[0] ^ (q[1] * 2654435761 & 0xFFFFFFFF) ^ (q[2] * 805459861 & 0xFFFFFFFF)) & (T - 1)
            wk = 1.0
            for a in range(3):
                wk = wk * (w[:, a] if (k >> a) & 1 else 1.0 - w[:, a])
            e = (l * T + h) * 2
            f = f + wk[:, None] * torch.stack([params[e], params[e + 1]], 1)
        feats.append(f)
    bins = (torch.arange(16, dtype=x9.dtype, device=dev) + 0.5) / 16.0
    for d in (x9[:, 3:6], x9[:, 6:9]):
        th = torch.acos(d[:, 2].clamp(-1.0, 1.0)) / math.pi
        ph = torch.atan2(d[:, 1], d[:, 0]) / (2 * math.pi) + 0.5
        feats += [torch.exp(-128.0 * (a[:, None] - bins) ** 2) for a in (th, ph)]
    return torch.cat(feats, 1)


def _exact_outputs(params, x9, log2_table):
    at = 32 * (1 << log2_table)
    a = _exact_encode(params, x9, log2_table)
    for l, (i, o) in enumerate(((96, 64), (64, 64), (64, 64), (64, 64), (64, 48))):
        w = params[at:at + i * o].reshape(o, i)
        at += i * o
        a = a @ w.T
        if l < 4:
            a = torch.relu(a)
    return a


def _exact_loss(o, omega, weight):
    """-sum(w / sum(w) log p(omega)) of the 8-lobe von Mises-Fisher mixture."""
    h = o[:, :40].reshape(-1, 8, 5)
    mu = h[..., :3] / h[..., :3].norm(dim=-1, keepdim=True).clamp_min(1e-6)
    lk = h[..., 3].clamp(-5.0, 7.0)
    k = torch.exp(lk)
    c = (mu * omega[:, None, :]).sum(-1)
    lp = torch.log_softmax(h[..., 4], -1) + lk - math.log(2 * math.pi) - torch.log(-torch.expm1(-2 * k)) + k * (c - 1.0)
    return -(weight / weight.sum() * torch.logsumexp(lp, -1)).sum()


def _exact_hits(c, seed):
    """Distance of the closest hit of each ray (its tmax where there is none), every triangle tested."""
    f = _scene(c, seed).flatten()
    v = torch.from_numpy(f.pos[f.idx.astype(np.int64)]).cuda().double()
    a, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    rays = torch.from_numpy(_rays(c, seed)).cuda().double()
    out = rays[:, 7].clone()
    for r0 in range(0, len(rays), 4096):
        r = rays[r0:r0 + 4096]
        o, d = r[:, None, :3], r[:, None, 4:7]
        p = torch.cross(d.expand(-1, len(a), -1), e2[None].expand(len(r), -1, -1), dim=-1)
        det = (p * e1).sum(-1)
        s = o - a
        u = (s * p).sum(-1) / det
        q = torch.cross(s, e1[None].expand(len(r), -1, -1), dim=-1)
        w = (q * d).sum(-1) / det
        t = (q * e2).sum(-1) / det
        hit = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > r[:, 3:4]) & (t < r[:, 7:8])
        out[r0:r0 + 4096] = torch.where(hit, t, r[:, 7:8]).min(1).values
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("forward", "gradient"):
        params, data = _network(c, seed)
        p, x = torch.from_numpy(params).cuda().double(), torch.from_numpy(data).cuda().double()
        if kind == "forward":
            return _exact_outputs(p, x, c["log2_table"])
        p.requires_grad_(True)
        loss = _exact_loss(_exact_outputs(p, x[:, :9], c["log2_table"]), x[:, 9:12], x[:, 12])
        loss.backward()
        return {"loss": float(loss), "grad": p.grad}
    if kind == "rays" and _triangles(c) * c["rays"] <= 2_000_000_000:
        return {"t": _exact_hits(c, seed), "prim": None, "b1": None, "b2": None, "occluded": None}
    # A path's course is decided by 32-bit comparisons: a film has no value of its own in 64 bits.
    return None
