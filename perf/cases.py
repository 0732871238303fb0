"""The measured work of the tracer: what a program that uses it calls, at the
sizes and with the options it uses.

Kinds of case:
  query  ray queries on a resident tree (BVH.trace_closest / BVH.trace_any)
  frame  a progressive accumulation: Params.reset, `frames` launch_kernels calls
         of one sample per pixel, one present
  build  a tree built on the GPU for geometry that has changed, then probed
  batch  many uneven render jobs in one Batch.run
  serve  render jobs and ray queries submitted to a Server and waited for

Scenes are the seeded ones of cudatracer_gb300/scenes.py. Queries, frames,
batches and served requests keep one resident scene and vary rays, cameras and
frame seeds; builds vary the geometry.
"""
import math

import numpy as np
import torch

from cudatracer_gb300 import api, scenes

_WORLD = {}  # resident context, scenes and trees, as a program keeps them
LIGHTS = ((-40.0, -40.0), (40.0, -40.0), (-40.0, 40.0), (40.0, 40.0))  # centres of the terrain's emissive quads, y = 70


def listed():
    return [
        # one 256x256 view of an 81,920-triangle model, on the reference's tree: a picking or
        # visibility query, where the latency of the call counts
        dict(name="closest_sphere_256", kind="query", scene="sphere", size=6, tree="reference", rays="pinhole",
             n=65536, any=False, eps=1e-12, tmax=20.0),
        # 4 M coherent rays against the same model on the tree built for traversal speed
        dict(name="closest_sphere_4m", kind="query", scene="sphere", size=6, tree="fast", rays="pinhole", n=4194304,
             any=False, eps=1e-12, tmax=1e34),
        # an odd number of shadow rays over a 727k-triangle terrain (visibility to area lights)
        dict(name="any_terrain_1m", kind="query", scene="terrain", size=512, tree="fast", rays="shadow", n=1000003,
             any=True, eps=1e-3, tmax=1e34),
        # incoherent rays through a triangle soup, answered as FP64 would (the precision path)
        dict(name="closest_soup_wide_4m", kind="query", scene="soup", size=4000000, tree="wide", rays="incoherent",
             n=4000000, any=False, eps=1e-12, tmax=1e34),
        # the smallest frame: one sample of a thumbnail after each camera move
        dict(name="frame_64x48", kind="frame", scene="terrain", size=64, tree="fast", width=64, height=48, depth=5,
             frames=1, math=2, shading=0, filter=0),
        # bit-exact frames on the reference's tree, odd width
        dict(name="frame_exact_641x360", kind="frame", scene="terrain", size=256, tree="reference", width=641,
             height=360, depth=8, frames=4, math=1, shading=0, filter=0),
        # the headline workload: 1920x1080, depth 8, 3.1 M triangles, exact shading, fast traversal
        dict(name="frame_1080p", kind="frame", scene="terrain", size=1024, tree="fast", width=1920, height=1080,
             depth=8, frames=16, math=2, shading=0, filter=0),
        # every material type with MIS, textures with bilinear filtering, CUDA's float functions
        dict(name="frame_full_960x540", kind="frame", scene="zoo", size=512, tree="fast", width=960, height=540,
             depth=8, frames=8, math=0, shading=1, filter=1),
        # a small deforming model rebuilt and probed (the reference's tree)
        dict(name="build_reference_20k", kind="build", scene="sphere", size=5, tree="reference", n=4096),
        # a large terrain rebuilt and probed (the tree for traversal speed)
        dict(name="build_fast_1m5", kind="build", scene="terrain", size=768, tree="fast", n=65536),
        # 24 uneven jobs (64..512 pixels a side, 1..16 samples, depth 4..12) in one batch
        dict(name="batch_24", kind="batch", jobs=24, side=512, spp=16, math=2),
        # requests in flight together: render jobs on terrains and closest-hit queries on a wide tree
        dict(name="serve_16", kind="serve", requests=16, side=384, spp=8, n=400000, math=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "frame", "frame", "frame", "build", "batch", "serve"])
    if kind == "query":
        scene = rng.choice(["sphere", "terrain", "soup"])
        size = {"sphere": rng.randint(3, 6), "terrain": int(_log(rng, 48, 900)), "soup": int(_log(rng, 5e3, 4e6))}[scene]
        rays = rng.choice({"sphere": ["pinhole", "incoherent"], "terrain": ["pinhole", "shadow", "incoherent"],
                           "soup": ["incoherent"]}[scene])
        tree = rng.choice(["reference", "fast", "wide"])
        if scene == "soup" and tree == "reference":
            tree = "fast"  # the reference's padded boxes swallow a soup's triangles
        return dict(kind=kind, scene=scene, size=size, tree=tree, rays=rays, n=int(_log(rng, 4096, 4.2e6)),
                    any=rays == "shadow" or rng.random() < 0.3, eps=1e-3 if scene == "terrain" else 1e-12,
                    tmax=rng.choice([1e34, 20.0]))
    if kind == "frame":
        w = int(_log(rng, 48, 1920))
        h = max(32, int(w * rng.uniform(0.45, 1.1)))
        h = min(h, 1080)
        mode = rng.choice([0, 1, 2, 2])
        frames = max(1, min(int(_log(rng, 1, 24)), int(16 * 1920 * 1080 / (w * h))))
        scene = rng.choice(["terrain", "zoo"])
        return dict(kind=kind, scene=scene, size=int(_log(rng, 64, 1024)), tree="reference" if mode == 1 else "fast",
                    width=w, height=h, depth=rng.randint(3, 8), frames=frames if mode != 1 else min(frames, 8),
                    math=mode, shading=rng.choice([0, 0, 1]), filter=rng.choice([0, 1]))
    if kind == "build":
        scene = rng.choice(["sphere", "terrain", "soup"])
        size = {"sphere": rng.randint(3, 7), "terrain": int(_log(rng, 48, 900)), "soup": int(_log(rng, 5e3, 2e6))}[scene]
        tree = rng.choice(["reference", "fast", "wide"])
        if scene == "soup" and tree == "reference":
            tree = "wide"
        return dict(kind=kind, scene=scene, size=size, tree=tree, n=int(_log(rng, 4096, 65536)))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 24), side=int(_log(rng, 96, 512)), spp=rng.randint(1, 16),
                    math=rng.choice([0, 2, 2, 1]))
    return dict(kind=kind, requests=rng.randint(2, 16), side=int(_log(rng, 96, 512)), spp=rng.randint(1, 8),
                n=int(_log(rng, 1e4, 1e6)), math=rng.choice([0, 2]))


# ---------------------------------------------------------------- scenes
def _ctx():
    if "ctx" not in _WORLD:
        _WORLD["ctx"] = api.Context(0)
    return _WORLD["ctx"]


def _host_scene(scene, size):
    """(scenes.Scene, camera) of a seeded scene."""
    key = ("host", scene, size)
    if key not in _WORLD:
        if scene == "sphere":
            got = scenes.sphere_scene(size), dict(position=(0.0, 0.0, 3.0), forward=(0.0, 0.0, -1.0),
                                                  up=(0.0, 1.0, 0.0), fov=45.0)
        elif scene == "soup":
            got = scenes.soup_scene(size), dict(position=(0.5, 0.5, 2.0), forward=(0.0, 0.0, -1.0),
                                                up=(0.0, 1.0, 0.0), fov=60.0)
        elif scene == "zoo":
            got = scenes.material_zoo_scene(grid=size, spheres=27, ground_textures=(256, 128))
        else:
            got = scenes.terrain_scene(grid=size, spheres=max(4, min(200, size // 5)))
        _WORLD[key] = got
    return _WORLD[key]


def _scene(scene, size):
    key = ("scene", scene, size)
    if key not in _WORLD:
        s, cam = _host_scene(scene, size)
        _WORLD[key] = _ctx().scene(scenes.scene_arrays(s), [api.Material(**m) for m in s.materials], s.textures,
                                   s.skybox_texture), cam
    return _WORLD[key]


def _build(sc, tree):
    return {"reference": sc.build_bvh_device, "fast": sc.build_bvh_fast_device, "wide": sc.build_bvh_wide}[tree]()


def _tree(scene, size, tree):
    key = ("tree", scene, size, tree)
    if key not in _WORLD:
        _WORLD[key] = _build(_scene(scene, size)[0], tree)
    return _WORLD[key]


def _triangles(scene, size):
    if scene == "sphere":
        return 20 * 4 ** size
    if scene == "soup":
        return size
    return 2 * (size - 1) ** 2 + (27 if scene == "zoo" else max(4, min(200, size // 5))) * 5120 + 8


# ---------------------------------------------------------------- rays (on the GPU, from the seed)
def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _rays(scene, size, rays, n, tmax, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    o = torch.zeros(n, 4, dtype=torch.float32, device="cuda")
    d = torch.empty(n, 4, dtype=torch.float32, device="cuda")
    if rays == "pinhole":  # a view through n pixel centres in scan order, the camera turned a little by the seed
        _, cam = _host_scene(scene, size)
        side = max(1, int(math.isqrt(n)))
        i = torch.arange(n, device="cuda")
        x = ((i % side) + 0.5) / side * 2 - 1
        y = 1 - ((i // side) + 0.5) / max(1, -(-n // side)) * 2
        turn = (rand(2) - 0.5) * 0.1
        w = torch.tensor(cam["forward"], dtype=torch.float64, device="cuda")
        w = w / w.norm()
        up = torch.tensor(cam["up"], dtype=torch.float64, device="cuda")
        u = torch.linalg.cross(w, up)
        u = u / u.norm()
        v = torch.linalg.cross(u, w)
        k = math.tan(math.radians(cam["fov"]) / 2)
        dirs = w + (x.double() * k + turn[0])[:, None] * u + (y.double() * k + turn[1])[:, None] * v
        o[:, :3] = torch.tensor(cam["position"], dtype=torch.float32, device="cuda")
        d[:, :3] = _unit(dirs).float()
        d[:, 3] = tmax
    elif rays == "shadow":  # from points over the terrain to points on its four lights
        p = torch.empty(n, 3, dtype=torch.float64, device="cuda")
        p[:, 0::2] = (rand(n, 2) - 0.5) * 160.0
        p[:, 1] = rand(n) * 20.0
        which = torch.randint(0, 4, (n,), generator=g, device="cuda")
        q = torch.empty_like(p)
        q[:, 0::2] = torch.tensor(LIGHTS, dtype=torch.float64, device="cuda")[which] + (rand(n, 2) - 0.5) * 12.0
        q[:, 1] = 70.0
        o[:, :3] = p.float()
        L = q - p
        d[:, :3] = _unit(L).float()
        d[:, 3] = (L.norm(dim=1) - 1e-3).float()
    else:  # origins all over the scene's box, directions all over the sphere
        s, _ = _host_scene(scene, size)
        lo = torch.from_numpy(s.vertices.min(0)).cuda().double()
        hi = torch.from_numpy(s.vertices.max(0)).cuda().double()
        o[:, :3] = (lo + rand(n, 3) * (hi - lo)).float()
        d[:, :3] = _unit(torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)).float()
        d[:, 3] = tmax
    return o, d


# ---------------------------------------------------------------- states
def _deform(v, seed):
    """Vertices moved along seeded waves of 2 % of the model's size."""
    rng = np.random.default_rng(int(seed))
    k = (2 * math.pi * rng.uniform(0.5, 2.0, 3)).astype(np.float32)
    shift = rng.uniform(0, 2 * math.pi, 3).astype(np.float32)
    span = np.float32(np.ptp(v, axis=0).max())
    return (v + np.float32(0.02) * span * np.sin((v[:, [1, 2, 0]] / span) * k + shift)).astype(np.float32)


class _Deformed:
    """A scene whose vertices moved a little: new geometry for a build."""

    def __init__(self, scene, size, seed):
        s, _ = _host_scene(scene, size)
        arrays = dict(scenes.scene_arrays(s), vertices=_deform(s.vertices, seed))
        self.scene = _ctx().scene(arrays, [api.Material(**m) for m in s.materials], s.textures, s.skybox_texture)

    def __del__(self):
        try:
            self.scene.close()
        except Exception:
            pass


def _job(rng, sizes, side, spp, mode, k, uneven=True):
    size = sizes[k % len(sizes)]
    sc, cam = _scene("terrain", size)
    s = int(_log_np(rng, 64, side)) if uneven else side
    p = api.default_params(s, s)
    p.max_depth = int(rng.integers(4, 13))
    p.frame_index = int(rng.integers(0, 1000)) * 2
    p.exact_math = mode
    return dict(scene=sc, bvh=_tree("terrain", size, "reference" if mode == 1 else "fast"), params=p,
                spp=max(1, int(_log_np(rng, 1, spp + 1))),
                camera=api.Camera(s, s, cam["fov"], cam["position"], cam["forward"], cam["up"]))


def _log_np(rng, lo, hi):
    return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))


def _shapes(case):
    """The uneven jobs' sizes come from the case alone, so that every seed asks for the same work."""
    return np.random.default_rng(97 + int(case.get("jobs", case.get("requests", 0))))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "query":
        tree = _tree(case["scene"], case["size"], case["tree"])
        o, d = _rays(case["scene"], case["size"], case["rays"], case["n"], case["tmax"], seed)
        st = dict(case=case, tree=tree, o=o, d=d)
        if case["any"]:
            st["occ"] = torch.empty(case["n"], dtype=torch.uint8, device="cuda")
        else:
            st["hit"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
            st["t"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
        return st
    if kind == "frame":
        sc, cam = _scene(case["scene"], case["size"])
        rng = np.random.default_rng(int(seed))
        turn = rng.uniform(-0.05, 0.05, 3)
        f = np.asarray(cam["forward"], np.float64) + turn
        f /= np.linalg.norm(f)
        w, h = case["width"], case["height"]
        camera = api.Camera(w, h, cam["fov"], cam["position"], tuple(float(x) for x in f), cam["up"])
        params = api.Params(w, h, camera=camera, max_depth=case["depth"], exact_math=case["math"],
                            shading_mode=case["shading"], texture_filter=case["filter"])
        return dict(case=case, scene=sc, tree=_tree(case["scene"], case["size"], case["tree"]), params=params,
                    job=api.RenderJob(_ctx(), w, h), first=2 * int(rng.integers(0, 100000)),
                    image=torch.empty(h * w, 4, dtype=torch.float32, device="cuda"))
    if kind == "build":
        o, d = _rays(case["scene"], case["size"], "incoherent", case["n"], 1e4, seed)
        return dict(case=case, held=_Deformed(case["scene"], case["size"], seed), o=o, d=d,
                    hit=torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                    t=torch.empty(case["n"], dtype=torch.float32, device="cuda"))
    rng = _shapes(case)
    if kind == "batch":
        jobs = [_job(rng, (128, 384, 512), case["side"], case["spp"], case["math"], k) for k in range(case["jobs"])]
        for j in jobs:
            j["params"].frame_index += 2 * (int(seed) % 1000003)
        return dict(case=case, batch=api.Batch(_ctx(), jobs, exact_math=case["math"]), jobs=len(jobs))
    jobs, rays = [], []
    for k in range(case["requests"]):
        if k % 2 == 0:
            j = _job(rng, (128, 384, 512), case["side"], case["spp"], case["math"], k)
            j["params"].frame_index += 2 * (int(seed) % 1000003)
            jobs.append(j)
        else:
            n = max(1, int(_log_np(rng, min(1e4, case["n"]), case["n"] + 1)))
            o, d = _rays("soup", 1000000, "incoherent", n, 1e34, int(seed) + k)
            rays.append((o.cpu().numpy(), d.cpu().numpy()))
    if "server" not in _WORLD:
        _WORLD["server"] = {}
    if case["math"] not in _WORLD["server"]:  # a resident server
        _WORLD["server"][case["math"]] = api.Server(_ctx(), hbm_budget=20 << 30, max_inflight_pixels=1 << 22,
                                                    exact_math=case["math"])
    return dict(case=case, server=_WORLD["server"][case["math"]], jobs=jobs, rays=rays,
                tree=_tree("soup", 1000000, "wide"))


def _view(tensor, owner):
    tensor.owner = owner  # a view of the library's memory: its owner lives as long
    return tensor


def run(state):
    kind = state["case"]["kind"]
    if kind == "query":
        c = state["case"]
        if c["any"]:
            return dict(occluded=state["tree"].trace_any(state["o"], state["d"], state["occ"], tri_eps=c["eps"]))
        hit, t = state["tree"].trace_closest(state["o"], state["d"], state["hit"], state["t"], tri_eps=c["eps"])
        return dict(hit=hit, t=t)
    if kind == "frame":
        p, job = state["params"], state["job"]
        p.reset(job)
        p.samples = state["first"]
        n = state["case"]["frames"]
        for _ in range(n):
            api.launch_kernels(job, state["scene"], state["tree"], p)
        job.present(2.0 * n, state["image"])
        return dict(accum=_view(job.accum_tensor(), job), image=state["image"])
    if kind == "build":
        tree = _build(state["held"].scene, state["case"]["tree"])
        hit, t = tree.trace_closest(state["o"], state["d"], state["hit"], state["t"], tri_eps=1e-12)
        info = tree.info()
        tree.close()
        return dict(hit=hit, t=t, nodes=info["quad_node_count"], depth=info["quad_depth"])
    if kind == "batch":
        state["batch"].run()
        return [_view(state["batch"].accum_tensor(k), state["batch"]) for k in range(state["jobs"])]
    srv = state["server"]
    ids = []
    for k in range(max(len(state["jobs"]), len(state["rays"]))):
        if k < len(state["jobs"]):
            ids.append(srv.submit_render(state["jobs"][k]))
        if k < len(state["rays"]):
            ids.append(srv.submit_query(state["tree"], *state["rays"][k]))
    return [srv.wait(i)[1] for i in ids]


# ---------------------------------------------------------------- what a pass cannot do without
def _per_ray(triangles):
    """(node visits, triangle tests) a ray needs at least: one four-wide path to a leaf of two triangles."""
    return max(1.0, math.log(max(2.0, triangles / 2), 4)), 2.0


def _trace_work(triangles, rays, out_bytes):
    v, t = _per_ray(triangles)
    tree = triangles * (48 + 27)  # triangle records, and four-wide nodes over leaves of two
    touched = min(tree, rays * (v * 128 + t * 48))
    return rays * (32 + out_bytes) + touched, rays * (v * 4 * 12 + t * 40)


def work(case):
    kind = case["kind"]
    if kind == "query":
        b, f = _trace_work(_triangles(case["scene"], case["size"]), case["n"], 1 if case["any"] else 8)
        return dict(bytes=b, flops=f)
    if kind == "build":
        n = _triangles(case["scene"], case["size"])
        # vertices and indices in, nodes (reference and traversal layout) and triangle records out
        b, f = _trace_work(n, case["n"], 8)
        return dict(bytes=n * (3 * 16 + 16) + n * (27 * 2 + 48 + 4) + b, flops=n * math.log2(max(2, n)) * 20 + f)
    if kind == "frame":
        px, n = case["width"] * case["height"], _triangles(case["scene"], case["size"])
        samples = px * case["frames"]
        # about two rays a sample; the scene once, the accumulation in and out, the image out
        v, t = _per_ray(n)
        touched = min(n * (48 + 27 + 128), samples * 2 * (v * 128 + t * 48 + 128))
        return dict(bytes=touched + px * 16 * 4, flops=samples * 2 * (v * 48 + t * 40 + 200))
    rng = _shapes(case)
    total = dict(bytes=0.0, flops=0.0)
    sizes = (128, 384, 512)
    for k in range(case.get("jobs", case.get("requests", 0))):
        if kind == "batch" or k % 2 == 0:
            side = int(_log_np(rng, 64, case["side"]))
            rng.integers(4, 13), rng.integers(0, 1000)
            spp = max(1, int(_log_np(rng, 1, case["spp"] + 1)))
            w = work(dict(kind="frame", scene="terrain", size=sizes[k % 3], width=side, height=side, frames=spp))
        else:
            n = max(1, int(_log_np(rng, min(1e4, case["n"]), case["n"] + 1)))
            w = work(dict(kind="query", scene="soup", size=1000000, n=n, any=False))
        total = {x: total[x] + w[x] for x in total}
    return total


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """Closest-hit distances by Moller-Trumbore over every triangle in binary64, where that is affordable.
    Frames, batches and served renders have none: a path's later bounces depend on every rounding before them."""
    n = case.get("n", 0)
    if case["kind"] not in ("query", "build") or case.get("any") or case["scene"] == "soup":
        return None
    if n * _triangles(case["scene"], case["size"]) > 6e9:
        return None
    s, _ = _host_scene(case["scene"], case["size"])
    verts, idx = s.vertices, s.indices
    if case["kind"] == "query":
        o, d = _rays(case["scene"], case["size"], case["rays"], n, case["tmax"], seed)
    else:
        verts = _deform(verts, seed)
        o, d = _rays(case["scene"], case["size"], "incoherent", n, 1e4, seed)
    v = torch.from_numpy(verts).cuda().double()
    ix = torch.from_numpy(idx.astype(np.int64)).cuda()
    p0 = v[ix[:, 0]]
    e1, e2 = v[ix[:, 1]] - p0, v[ix[:, 2]] - p0
    nrm = torch.linalg.cross(e1, e2)
    # the triple products of all rays and triangles as matrix products, with m = o x d:
    #   t = (p0 - o) . n / d . n,  u = -(m . e2 + d . (p0 x e2)) / d . n,  w = (m . e1 + d . (p0 x e1)) / d . n
    ox, dx = o[:, :3].double(), d[:, :3].double()
    best = d[:, 3].double().clone()
    m = torch.linalg.cross(ox, dx)
    a2, a1 = torch.linalg.cross(p0, e2), torch.linalg.cross(p0, e1)
    pn = (p0 * nrm).sum(1)
    block = max(1, int(4e7 // max(1, n)))
    for b in range(0, ix.shape[0], block):
        sl = slice(b, b + block)
        det = dx @ nrm[sl].T
        u = -(m @ e2[sl].T + dx @ a2[sl].T)
        w = m @ e1[sl].T + dx @ a1[sl].T
        t = (pn[sl] - ox @ nrm[sl].T) / det
        u, w = u / det, w / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0)
        best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, math.inf)).amin(1))
    out = dict(hit=None, t=best)
    if case["kind"] == "build":
        out.update(nodes=None, depth=None)
    return out
