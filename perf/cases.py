"""Timed cases: ray queries, renders and store builds through the public entry
points (`cgspline_gb300.rt`), over the sizes that the tests and bench.py use.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
a case's inputs from a seed, run() is one pass, work() the bytes and operations
that a pass cannot do without, exact() the results in float64 by plain torch:
patches that a ray's box test keeps, Newton from a grid of seeds on each, the
nearest root."""
import math

import numpy as np
import torch

from cgspline_gb300 import rt, scenes

FAR = 100.0  # ray extent of the queries: a far plane behind every scene here
LEVEL = {"fp32": rt.FP32, "polish": rt.FP32_POLISH64, "graze": rt.FP32_GRAZE64}
SPLIT = {"reference": rt.SPLIT_REFERENCE, "mirror": rt.SPLIT_MIRROR}
METHOD = {"clip": rt.CLIP, "subdiv": rt.SUBDIV}


def listed():
    return [
        # the pick under a mouse cursor and its neighbourhood: a few rays from host memory
        {"name": "pick", "kind": "pick", "objects": 12, "patches": 1500, "n": 33, "level": "polish"},
        # primary rays of the full frame, asked for as a query (depth, object id and uv buffers)
        {"name": "primary", "kind": "closest", "scene": "torus", "patches": 16384, "split": "reference", "rays": "camera",
         "n": 2073600, "level": "polish", "method": "clip"},
        # scattered rays (gathers, ambient occlusion with distances) through a large union scene
        {"name": "scattered", "kind": "closest", "scene": "union", "objects": 40, "patches": 60000, "split": "mirror",
         "rays": "scattered", "n": 301111, "level": "fp32", "method": "clip"},
        # shadow rays from points of a surface to a light
        {"name": "shadow", "kind": "shadow", "patches": 16384, "split": "reference", "n": 640001, "level": "fp32",
         "method": "clip"},
        # the other intersector
        {"name": "subdivide", "kind": "closest", "scene": "torus", "patches": 2048, "split": "reference", "rays": "camera",
         "n": 131101, "level": "fp32", "method": "subdiv"},
        # silhouette rays at the full precision form
        {"name": "grazing", "kind": "closest", "scene": "torus", "patches": 16384, "split": "reference", "rays": "grazing",
         "n": 65537, "level": "graze", "method": "clip"},
        # the full frame: 1080p, one mirror bounce, PBR, shadow rays, into pinned host memory
        {"name": "frame", "kind": "frame", "scene": "torus", "patches": 16384, "split": "reference", "width": 1920,
         "height": 1080, "depth": 1, "level": "polish", "sampling": "mirror"},
        # a thumbnail or an interactive preview: a small odd frame with sampled bounces
        {"name": "preview", "kind": "frame", "scene": "union", "objects": 10, "patches": 3000, "split": "reference",
         "width": 319, "height": 181, "depth": 3, "level": "fp32", "sampling": "monte-carlo"},
        # render requests of several scenes, sizes and sample counts in one wavefront
        {"name": "batch", "kind": "batch", "groups": 8, "objects": 16, "patches": 8000, "split": "reference",
         "requests": 12, "side": 512, "depth": 1, "level": "polish"},
        # explicit (ray, patch) pairs and the normals at their roots
        {"name": "pairs", "kind": "pairs", "patches": 8192, "n": 200003, "method": "clip"},
        # the perfect hash of one large surface's BVH
        {"name": "hash", "kind": "hash", "leaves": 20000},
        # a scene made resident: BVHs, upload, perfect hashes, its tables read back
        {"name": "store", "kind": "store", "objects": 24, "patches": 30000, "split": "reference"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "closest", "closest", "closest", "shadow", "frame", "batch", "pairs", "hash", "store"])
    split = rng.choice(["reference", "reference", "mirror"])
    method = rng.choice(["clip", "clip", "subdiv"])
    level = rng.choice(["fp32", "polish", "polish"])
    if kind == "pick":
        return {"kind": kind, "objects": rng.randint(1, 24), "patches": _log(rng, 500, 20000), "n": _log(rng, 1, 2000),
                "level": level}
    if kind == "closest":
        rays = rng.choice(["camera", "camera", "scattered", "grazing"])
        n = _log(rng, 1000, 1500000 if rays == "camera" else 200000)
        if rays == "grazing":
            method, level, n = "clip", "graze", min(n, 65000)
        elif method == "subdiv":
            n, level = min(n, 200000), "fp32"
        case = {"kind": kind, "scene": rng.choice(["torus", "union"]), "patches": _log(rng, 256, 60000), "split": split,
                "rays": rays, "n": n, "level": level, "method": method}
        if case["scene"] == "union":
            case["objects"] = rng.randint(2, 48)
        return case
    if kind == "shadow":
        return {"kind": kind, "patches": _log(rng, 500, 30000), "split": split, "n": _log(rng, 1000, 600000),
                "level": "fp32", "method": method if rng.random() < 0.3 else "clip"}
    if kind == "frame":
        w = _log(rng, 65, 1600)
        case = {"kind": kind, "scene": rng.choice(["torus", "union"]), "patches": _log(rng, 256, 20000), "split": split,
                "width": w, "height": max(33, w * rng.randint(40, 60) // 90), "depth": rng.randint(0, 3), "level": level,
                "sampling": rng.choice(["mirror", "monte-carlo"])}
        if case["scene"] == "union":
            case["objects"] = rng.randint(2, 30)
        return case
    if kind == "batch":
        return {"kind": kind, "groups": rng.randint(2, 8), "objects": rng.randint(4, 16), "patches": _log(rng, 500, 8000),
                "split": split, "requests": rng.randint(2, 12), "side": _log(rng, 64, 500), "depth": rng.randint(0, 2),
                "level": level}
    if kind == "pairs":
        return {"kind": kind, "patches": _log(rng, 128, 16384), "n": _log(rng, 500, 300000), "method": method}
    if kind == "hash":
        return {"kind": kind, "leaves": _log(rng, 64, 30000)}
    return {"kind": kind, "objects": rng.randint(1, 40), "patches": _log(rng, 500, 40000), "split": split}


# ------------------------------------------------------------------ inputs --
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _hashable(n, bad, lo):
    """The next grid size at or below n whose BVH the perfect hash takes."""
    while n > lo and n in bad:
        n -= 1
    return n


def _torus_scene(patches, seed):
    nv = _hashable(max(3, int(math.sqrt(patches / 2.0) + 0.5)), scenes.TORUS_NV_NO_HASH, 3)
    nu = 2 * nv
    if patches == 16384:
        nu = nv = 128
    sc = scenes.scene_c2(seed % 1000003, nu=nu, nv=nv)
    return sc


def _union_scene(objects, patches, seed):
    """Spheres and tori of fixed sizes at seeded places, each displaced by its own seed."""
    r = np.random.RandomState(seed % (1 << 31))
    weight = np.array([0.4 + (k * 7 % 11) / 5.0 for k in range(objects)])
    per = patches * weight / weight.sum()
    surfaces, obs = [], []
    for k in range(objects):
        if k % 2 == 0:
            n = _hashable(max(1, int(math.sqrt(per[k] / 6.0) + 0.5)), scenes.SPHERE_N_NO_HASH, 1)
            s = scenes.cube_sphere_surface(1.0, n, 0.03, int(r.randint(1 << 30)))
        else:
            n = _hashable(max(3, int(math.sqrt(per[k] / 2.0) + 0.5)), scenes.TORUS_NV_NO_HASH, 3)
            s = scenes.torus_surface(1.0, 0.35, 2 * n, n, 0.02, int(r.randint(1 << 30)))
        q = r.randn(4)
        x, y, z, w = q / np.sqrt(q @ q)
        R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                      [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                      [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
        scale, pos = 0.5 + r.rand(), r.uniform(-4.0, 4.0, 3)
        M, W = np.eye(4), np.eye(4)
        M[:3, :3], M[:3, 3] = R * scale, pos
        W[:3, :3], W[:3, 3] = R.T / scale, -(R.T / scale) @ pos
        metal = float(r.rand() < 0.4)
        mat = scenes.Material(tuple(float(v) for v in r.uniform(0.3, 0.9, 3)), (0.9, 0.85, 0.8) if metal else (0.04,) * 3,
                              metal, float(r.uniform(0.1, 0.9)))
        surfaces.append(s)
        obs.append(scenes.Object(k, M.T.reshape(16).astype(np.float32), W.T.reshape(16).astype(np.float32), mat))
    lights = [scenes.Light((120.0,) * 3, 1.0, tuple(float(v) for v in 14.0 * d / np.sqrt(d @ d)), 0.0, (0.0, 0.0, -1.0), math.pi)
              for d in r.randn(2, 3)]
    return scenes.Scene(surfaces, obs, lights, name="union")


def _scene(case, seed):
    if case.get("scene") == "torus" or case["kind"] in ("shadow", "pairs"):
        return _torus_scene(case["patches"], seed)
    return _union_scene(case["objects"], case["patches"], seed)


def _view(case, seed):
    """(eye, target, vertical field of view) for the case's scene, moved a little by the seed."""
    r = np.random.RandomState((seed + 77) % (1 << 31))
    if case.get("scene") == "torus":
        return np.array([2.0, -5.0, 8.0]) + r.uniform(-0.3, 0.3, 3), np.array([0.0, 0.0, -0.5]), math.radians(55.0)
    d = r.randn(3)
    return 13.0 * d / np.sqrt(d @ d), np.zeros(3), math.radians(50.0)


def _camera(case, seed):
    eye, target, fovy = _view(case, seed)
    return scenes.Camera(scenes.look_at(eye, target, (0.0, 0.0, 1.0) if abs(eye[2]) < 12.0 else (0.0, 1.0, 0.0)),
                         tuple(float(np.float32(v)) for v in eye), (1, 1, 1), float(np.float32(fovy)))


def _camera_rays(case, seed, n, device):
    """The first n pixels' rays of a 16:9 image of at least n pixels, scanline order."""
    eye, target, fovy = _view(case, seed)
    h = max(1, int(math.sqrt(n * 9.0 / 16.0)))
    w = -(-n // h)
    f = target - eye
    f = f / np.sqrt(f @ f)
    s = np.cross(f, [0.0, 0.0, 1.0] if abs(f[2]) < 0.95 else [0.0, 1.0, 0.0])
    s = s / np.sqrt(s @ s)
    u = np.cross(s, f)
    f, s, u, eye = (torch.tensor(v, dtype=torch.float64, device=device)[:, None] for v in (f, s, u, eye))
    k = torch.arange(n, device=device)
    th = math.tan(0.5 * fovy)
    x = ((k % w).double() + 0.5) / w * 2 - 1
    y = 1 - ((k // w).double() + 0.5) / h * 2
    d = f + (x * (th * w / h)) * s + (y * th) * u
    d = d / d.norm(dim=0, keepdim=True)
    return torch.cat([eye.expand(3, n), d, torch.full((1, n), FAR, dtype=torch.float64, device=device)]).float().contiguous()


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed % (1 << 62))
    return g


def _scattered_rays(seed, n, device):
    g = _generator(seed + 5, device)
    o = torch.rand((3, n), generator=g, device=device, dtype=torch.float64) * 10 - 5
    d = torch.randn((3, n), generator=g, device=device, dtype=torch.float64)
    d = d / d.norm(dim=0, keepdim=True)
    return torch.cat([o, d, torch.full((1, n), FAR, dtype=torch.float64, device=device)]).float().contiguous()


def _grazing_rays(scene, seed, n, device):
    rays = torch.from_numpy(scenes.grazing_rays(scene.surfaces[-1], n, seed=seed % 1000003)).to(device)
    rays[6] = 12.0  # the rays start at most 10 units before their surface point
    ob = scene.objects[-1]
    m = torch.from_numpy(ob.local2world.astype(np.float64).reshape(4, 4).T.copy()).to(device)
    o = m[:3, :3] @ rays[0:3].double() + m[:3, 3:]
    d = m[:3, :3] @ rays[3:6].double()
    return torch.cat([o, d / d.norm(dim=0, keepdim=True), rays[6:].double()]).float().contiguous()


def _rays(case, scene, seed, device):
    if case["rays"] == "camera":
        return _camera_rays(case, seed, case["n"], device)
    if case["rays"] == "scattered":
        return _scattered_rays(seed, case["n"], device)
    return _grazing_rays(scene, seed, case["n"], device)


def _eval(nets, u, v):
    """Points and partials of nets (m, 4 [j], 4 [i], c) at (u, v), both (m, ...)."""
    def b(t):
        s = 1 - t
        return torch.stack([s * s * s, 3 * t * s * s, 3 * t * t * s, t * t * t], -1)

    def db(t):
        s = 1 - t
        return torch.stack([-3 * s * s, 3 * s * s - 6 * t * s, 6 * t * s - 3 * t * t, 3 * t * t], -1)

    bu, bv, du, dv = b(u), b(v), db(u), db(v)
    ru = torch.einsum("m...i,mjic->m...jc", bu, nets)
    rd = torch.einsum("m...i,mjic->m...jc", du, nets)
    return (torch.einsum("m...j,m...jc->m...c", bv, ru), torch.einsum("m...j,m...jc->m...c", bv, rd),
            torch.einsum("m...j,m...jc->m...c", dv, ru))


def _nets(scene, device):
    """World-space nets (P, 4, 4, 3) in float64, their object and their patch within it."""
    nets, obj, pid = [], [], []
    for k, ob in enumerate(scene.objects):
        p = torch.from_numpy(scene.surfaces[ob.surface].patches().astype(np.float64)).to(device)
        back = torch.from_numpy(ob.world2local.astype(np.float64).reshape(4, 4).T.copy()).to(device)
        q = p @ torch.linalg.inv(back).T
        nets.append((q[..., :3] / q[..., 3:]).reshape(-1, 4, 4, 3))
        obj.append(torch.full((p.shape[0],), k, device=device))
        pid.append(torch.arange(p.shape[0], device=device))
    return torch.cat(nets), torch.cat(obj), torch.cat(pid)


def _surface_points(scene, seed, n, device):
    """n seeded points of the scene's first surface, in patch order, with normals, patch and (u, v)."""
    nets = torch.from_numpy(scene.surfaces[0].patches()[..., :3].astype(np.float64)).to(device).reshape(-1, 4, 4, 3)
    g = _generator(seed + 9, device)
    p = torch.sort(torch.randint(nets.shape[0], (n,), generator=g, device=device)).values
    uv = torch.rand((2, n), generator=g, device=device, dtype=torch.float64)
    S, Su, Sv = _eval(nets[p], uv[0], uv[1])
    N = torch.linalg.cross(Su, Sv)
    return S, N / N.norm(dim=1, keepdim=True), p


def _shadow_rays(case, scene, seed, device):
    n = case["n"]
    S, N, _ = _surface_points(scene, seed, 3 * n + 64, device)
    r = np.random.RandomState((seed + 31) % (1 << 31))
    light = torch.tensor([6.0, -6.0, 8.0] + r.uniform(-1, 1, 3), dtype=torch.float64, device=device)
    L = light - S
    dist = L.norm(dim=1, keepdim=True)
    L = L / dist
    lit = torch.nonzero((N * L).sum(1) > 1e-3)[:, 0]
    at = lit[torch.arange(n, device=device) * lit.numel() // n]
    return torch.cat([(S + 1e-4 * L)[at].T, L[at].T, dist[at].T]).float().contiguous()


def _pairs(case, scene, seed, device):
    """Rays toward seeded points of seeded patches, a few of them past the patch's edge."""
    n = case["n"]
    S, N, p = _surface_points(scene, seed, n, device)
    g = _generator(seed + 13, device)
    a = torch.randn((n, 3), generator=g, device=device, dtype=torch.float64)
    d = -(N + 0.7 * a / a.norm(dim=1, keepdim=True))
    d = d / d.norm(dim=1, keepdim=True)
    o = S - (1.0 + 4.0 * torch.rand((n, 1), generator=g, device=device, dtype=torch.float64)) * d
    shift = torch.randint(scene.surfaces[0].patch_count, (n,), generator=g, device=device)
    q = torch.where(torch.rand(n, generator=g, device=device) < 0.15, shift, p)
    rays = torch.cat([o.T, d.T, torch.full((1, n), FAR, dtype=torch.float64, device=device)]).float().contiguous()
    return rays, q.to(torch.int32)


# --------------------------------------------------------------------- run --
def prepare(case, seed):
    kind = case["kind"]
    if kind == "hash":
        keys = scenes.bvh_keys(_hash_leaves(case["leaves"]))
        keys = keys[np.random.RandomState(seed % (1 << 31)).permutation(keys.size)]
        return {"case": case, "keys": torch.from_numpy(keys.view(np.int32)).cuda()}
    if kind == "store":
        return {"case": case, "scene": _scene(case, seed),
                "rays": _camera_rays(dict(case, scene="union"), seed, 4096, "cuda")}
    if kind == "batch":
        parts = [dict(case, scene="union", patches=max(300, case["patches"] >> (k % 4))) for k in range(case["groups"])]
        store = rt.GpuScene([_scene(c, seed + 100 * k) for k, c in enumerate(parts)], split=SPLIT[case["split"]])
        reqs = []
        for k in range(case["requests"]):
            g = k % case["groups"]
            side = max(33, case["side"] * (4 - k % 4) // 4 - k)
            reqs.append(rt.Request.alloc(g, _camera(parts[g], seed + k), side, max(17, side * 2 // 3), spp=1 + k % 3 * 2 % 4,
                                         linear=True))
        options = rt.Options(recursion_depth=case["depth"], precision=LEVEL[case["level"]])
        return {"case": case, "store": store, "requests": reqs, "tracer": rt.RayTracer(options)}
    scene = _scene(case, seed)
    store = rt.GpuScene(scene, split=SPLIT[case.get("split", "reference")])
    if kind == "pick":
        return {"case": case, "store": store,
                "rays": np.ascontiguousarray(_camera_rays(dict(case, scene="union"), seed, case["n"], "cpu").numpy())}
    if kind == "closest":
        return {"case": case, "store": store, "rays": _rays(case, scene, seed, "cuda")}
    if kind == "shadow":
        return {"case": case, "store": store, "rays": _shadow_rays(case, scene, seed, "cuda")}
    if kind == "pairs":
        rays, p = _pairs(case, scene, seed, "cuda")
        return {"case": case, "store": store, "rays": rays, "patch": p, "t": torch.full((case["n"],), FAR, device="cuda")}
    w, h = case["width"], case["height"]
    fb = torch.empty((h, w), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    lin = torch.empty((h, w, 3), dtype=torch.float32, pin_memory=True).numpy()
    options = rt.Options(recursion_depth=case["depth"], precision=LEVEL[case["level"]],
                         sampling=rt.MIRROR if case["sampling"] == "mirror" else rt.MONTE_CARLO)
    return {"case": case, "store": store, "camera": _camera(case, seed), "out": (fb, lin), "tracer": rt.RayTracer(options)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "pick":
        return state["store"].intersect(state["rays"], precision=LEVEL[case["level"]])
    if kind == "closest":
        return state["store"].intersect(state["rays"], method=METHOD[case["method"]], precision=LEVEL[case["level"]])
    if kind == "shadow":
        return {"occluded": state["store"].intersect(state["rays"], method=METHOD[case["method"]], any_hit=True)["patch"]}
    if kind == "frame":
        fb, lin = state["tracer"].render_host(state["camera"], state["store"], case["width"], case["height"], out=state["out"])
        return {"fb": fb.view(np.int32), "linear": lin}
    if kind == "batch":
        state["tracer"].render_batch(state["requests"], state["store"])
        torch.cuda.current_stream().synchronize()  # the store takes its next batch when this one is done
        return [[q.framebuffer, q.linear] for q in state["requests"]]
    if kind == "pairs":
        found, t, u, v = rt.do_bezier_clipping(state["store"], 0, state["rays"], state["patch"], t=state["t"],
                                               method=METHOD[case["method"]])
        return {"found": found, "t": t, "u": u, "v": v, "normal": rt.normal(state["store"], 0, state["patch"], u, v)}
    if kind == "hash":
        f = rt.PerfectHashFunction()
        status = f.build(state["keys"])
        return {"status": status, "params": [f.A, f.B, f.N, f.mask, f.trials], "disp": f.disp.view(np.int32),
                "table": f.table.view(np.int32)}
    store = rt.GpuScene(state["scene"], split=SPLIT[case["split"]])
    hits = store.intersect(state["rays"], precision=rt.FP32_POLISH64)
    out = [store.bvh(k) for k in [*range(store.surfaces), -1]]
    store.close()
    return {"hits": hits, **{k: np.concatenate([b[k].reshape(-1) for b in out]).view(np.int32)
                             for k in ("nodes", "keys", "indices", "table", "disp")}}


def _hash_leaves(leaves):
    """The next grid-like leaf count at or below `leaves` that the perfect hash takes."""
    nv = _hashable(max(3, int(math.sqrt(leaves / 2.0))), scenes.TORUS_NV_NO_HASH, 3)
    return 2 * nv * nv


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes: rays in, results out, the scene's control points once.  Operations: a box test a level of a balanced tree
    over the patches, one projected net and the mean clip iterations of a hit (4.5 on the torus frame's rays)."""
    kind, p = case["kind"], case.get("patches", 0)

    def rays(n):
        return n * (200 + 24 * math.log2(max(p, 2)) + 296 + 4.5 * 470)

    if kind == "hash":
        n = 2 * _hash_leaves(case["leaves"]) - 1
        return {"bytes": 4 * n + 4 * n + 2 * n, "flops": 6 * n}
    if kind == "store":
        return {"bytes": p * (256 + 2 * 64 + 2 * 4 * 3.5), "flops": p * (16 * 12 + 2 * 6)}
    if kind == "pairs":
        return {"bytes": case["n"] * (28 + 8 + 16 + 12 + 4) + min(p, case["n"]) * 256,
                "flops": case["n"] * (296 + 4.5 * 470 + 300)}
    if kind == "frame":
        n = case["width"] * case["height"]
        return {"bytes": n * 16 + min(p, n) * 256, "flops": rays(n) * 2}
    if kind == "batch":
        n = s = 0
        for k in range(case["requests"]):
            side = max(33, case["side"] * (4 - k % 4) // 4 - k)
            n += side * max(17, side * 2 // 3)
            s += side * max(17, side * 2 // 3) * (1 + k % 3 * 2 % 4)
        return {"bytes": n * 16 + p * 256 * case["groups"] // 2, "flops": rays(s) * 2}
    return {"bytes": case["n"] * (28 + (4 if kind == "shadow" else 20)) + min(p, case["n"]) * 256, "flops": rays(case["n"])}


# ------------------------------------------------------------------- exact --
def _roots(nets, o, d, seeds):
    """The nearest root in front of each pair's ray: nets (m, 4, 4, 3), o and d (m, 3).  t is inf where there is none."""
    e = torch.where(d[:, 2:].abs() < 0.9, torch.tensor([0.0, 0.0, 1.0], dtype=d.dtype, device=d.device),
                    torch.tensor([1.0, 0.0, 0.0], dtype=d.dtype, device=d.device))
    a = torch.linalg.cross(d, e)
    a = a / a.norm(dim=1, keepdim=True)
    b = torch.linalg.cross(d, a)
    b = b / b.norm(dim=1, keepdim=True)
    rel = nets - o[:, None, None]
    net = torch.stack([(rel * a[:, None, None]).sum(-1), (rel * b[:, None, None]).sum(-1)], -1)
    m = net.shape[0]
    g = (torch.arange(seeds, dtype=d.dtype, device=d.device) + 0.5) / seeds
    u = g.repeat(seeds).expand(m, -1).clone()
    v = g.repeat_interleave(seeds).expand(m, -1).clone()
    for _ in range(12):
        F, Fu, Fv = _eval(net, u, v)
        det = Fu[..., 0] * Fv[..., 1] - Fu[..., 1] * Fv[..., 0]
        det = torch.where(det.abs() < 1e-300, torch.full_like(det, 1e-300), det)
        du = (F[..., 0] * Fv[..., 1] - F[..., 1] * Fv[..., 0]) / det
        dv = (Fu[..., 0] * F[..., 1] - Fu[..., 1] * F[..., 0]) / det
        u = (u - du.clamp(-0.5, 0.5)).clamp(-0.2, 1.2)
        v = (v - dv.clamp(-0.5, 0.5)).clamp(-0.2, 1.2)
    F = _eval(net, u, v)[0]
    S = _eval(nets, u, v)[0] - o[:, None]
    t = (S * d[:, None]).sum(-1) / (d * d).sum(-1, keepdim=True)
    size = (net.amax((1, 2)) - net.amin((1, 2))).amax(-1, keepdim=True)
    ok = (F.norm(dim=-1) < 1e-9 * size) & (u > -1e-7) & (u < 1 + 1e-7) & (v > -1e-7) & (v < 1 + 1e-7) & (t > 0)
    t = torch.where(ok, t, torch.full_like(t, math.inf))
    t, k = t.min(dim=1)
    return t, u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]


def _slabs(lo, hi, o, inv):
    a, b = (lo - o) * inv, (hi - o) * inv
    return (torch.minimum(a, b).amax(-1) <= torch.maximum(a, b).amin(-1)) & (torch.maximum(a, b).amin(-1) > 0)


def _closest(scene, rays, seeds):
    """The nearest root of each ray over all patches: t (tmax on a miss), u, v (0 on a miss)."""
    dev = rays.device
    nets = _nets(scene, dev)[0]
    lo, hi = nets.amin((1, 2)), nets.amax((1, 2))
    c = (lo + hi) / 2
    grid = ((c - c.amin(0)) / (c.amax(0) - c.amin(0)).clamp(min=1e-9) * 15.999).long()
    code = sum(((grid[:, a] >> b) & 1) << (3 * b + a) for a in range(3) for b in range(4))
    order = torch.argsort(code)
    nets, lo, hi = nets[order], lo[order], hi[order]
    P, K = nets.shape[0], 32
    C = -(-P // K)
    pad = C * K - P
    blo = torch.cat([lo, lo[-1:].expand(pad, 3)]).reshape(C, K, 3).amin(1)
    bhi = torch.cat([hi, hi[-1:].expand(pad, 3)]).reshape(C, K, 3).amax(1)
    eps = 1e-5 * (hi.amax() - lo.amin())
    flo, fhi, blo, bhi = (lo - eps).float(), (hi + eps).float(), (blo - eps).float(), (bhi + eps).float()
    n = rays.shape[1]
    t, u, v = rays[6].double().clone(), torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
    step = max(256, min(65536, (1 << 27) // max(C, 1)))
    for r0 in range(0, n, step):
        o, d = rays[0:3, r0:r0 + step].T.contiguous(), rays[3:6, r0:r0 + step].T.contiguous()
        inv = 1 / torch.where(d.abs() < 1e-12, torch.full_like(d, 1e-12), d)
        ray, cl = torch.nonzero(_slabs(blo, bhi, o[:, None], inv[:, None]), as_tuple=True)
        pr, pp = [], []
        for q0 in range(0, ray.numel(), 1 << 20):
            rr, cc = ray[q0:q0 + (1 << 20)], cl[q0:q0 + (1 << 20)]
            ids = cc[:, None] * K + torch.arange(K, device=dev)
            keep = ids < P
            ids = ids.clamp(max=P - 1)
            a, b = torch.nonzero(_slabs(flo[ids], fhi[ids], o[rr][:, None], inv[rr][:, None]) & keep, as_tuple=True)
            pr.append(rr[a])
            pp.append(ids[a, b])
        if not pr:
            continue
        pr, pp = torch.cat(pr), torch.cat(pp)
        for q0 in range(0, pr.numel(), 1 << 17):
            rr, pi = pr[q0:q0 + (1 << 17)], pp[q0:q0 + (1 << 17)]
            tt, uu, vv = _roots(nets[pi], o[rr].double(), d[rr].double(), seeds)
            best = torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=dev).scatter_reduce(0, rr, tt, "amin")
            win = (tt == best[rr]) & (tt < t[r0 + rr])
            at = r0 + rr[win]
            t[at], u[at], v[at] = tt[win], uu[win], vv[win]
    return t, u, v


def exact(case, seed):
    dev, kind = _device(), case["kind"]
    if kind in ("shadow", "frame", "batch", "hash"):
        return None  # whole numbers, or an image of thousands of shaded rays a pixel row
    scene = _scene(case, seed)
    seeds = 6 if case.get("rays") == "grazing" else 3
    if kind == "pairs":
        rays, p = _pairs(case, scene, seed, dev)
        nets = torch.from_numpy(scene.surfaces[0].patches()[..., :3].astype(np.float64)).to(dev).reshape(-1, 4, 4, 3)
        n = case["n"]
        t = torch.full((n,), FAR, dtype=torch.float64, device=dev)
        u, v = torch.zeros_like(t), torch.zeros_like(t)
        for q in range(0, n, 1 << 17):
            k = slice(q, min(n, q + (1 << 17)))
            o, d = rays[0:3, k].T.double(), rays[3:6, k].T.double()
            tt, uu, vv = _roots(nets[p[k].long()], o, d, 4)
            hit = tt * d.norm(dim=1) < FAR
            t[k] = torch.where(hit, tt * d.norm(dim=1), t[k])
            u[k], v[k] = torch.where(hit, uu, u[k]), torch.where(hit, vv, v[k])
        _, Su, Sv = _eval(nets[p.long()], u, v)
        N = torch.linalg.cross(Su, Sv)
        return {"found": None, "t": t, "u": u, "v": v, "normal": (N / N.norm(dim=1, keepdim=True)).T.contiguous()}
    if kind == "pick":
        rays = _camera_rays(dict(case, scene="union"), seed, case["n"], "cpu").to(dev)
    elif kind == "store":
        rays = _camera_rays(dict(case, scene="union"), seed, 4096, dev)
    else:
        rays = _rays(case, scene, seed, dev)
    t, u, v = _closest(scene, rays, seeds)
    hits = {"t": t, "u": u, "v": v, "patch": None, "object": None}
    return hits if kind != "store" else {"hits": hits, "nodes": None, "keys": None, "indices": None, "table": None, "disp": None}
