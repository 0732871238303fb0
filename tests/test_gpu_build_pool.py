"""The pool of device builds: what it keeps is bounded, given back when it is wanted, and
a tree's memory is freed safely whoever destroys it and whatever runs meanwhile."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _scene(ctx, n, seed=1):
    from cudatracer_gb300 import api, scenes

    s = scenes.soup_scene(n, seed=seed)
    return ctx.scene({"vertices": s.vertices, "normals": s.normals, "indices": s.indices}, [api.Material()])


def _free():
    import torch

    torch.cuda.synchronize()
    gc.collect()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_trees_destroyed_through_another_context_leave_the_bound(lib):
    """1 GiB beyond live trees is what a pool may keep, also of trees that another context gave back."""
    from cudatracer_gb300 import api

    a, b = api.Context(0), api.Context(0)
    sc = _scene(a, 1000000)
    before = _free()
    trees = [sc.build_bvh_fast_device() for _ in range(16)]
    held = sum(t.info()["device_bytes"] for t in trees)
    assert held > 3 * GIB // 2
    for t in trees:
        assert b.lib.ct_bvh_destroy(b.h, t.h) == 0
        t.h = None
    assert before - _free() <= GIB + (128 << 20)
    sc.close()
    b.close()
    a.close()


KINDS = ("build_bvh_device", "build_bvh_fast_device", "build_bvh_wide")


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_destroy_while_a_graph_is_captured(gpu_ctx, kind, mode):
    """As for any cudaFree: in relaxed capture, or in another thread than a thread-local one."""
    import threading

    import torch

    sc = _scene(gpu_ctx, 3000)
    used = gpu_ctx.device_bytes
    tree = getattr(sc, kind)()
    x = torch.zeros(8, device="cuda")
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        g.capture_begin(capture_error_mode=mode)
        x.add_(1)
        if mode == "relaxed":
            tree.close()
        else:
            t = threading.Thread(target=tree.close)
            t.start()
            t.join()
        x.add_(1)
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8 and gpu_ctx.device_bytes == used
    sc.close()


@pytest.mark.parametrize("kind", ["build_bvh_device", "build_bvh_fast_device"])
def test_trees_closed_right_behind_their_queries(gpu_ctx, kind):
    """Queries in flight on a non-blocking stream when their tree is destroyed, while other
    threads build and destroy trees in the memory that it gives back."""
    import threading

    import torch

    from cudatracer_gb300 import scenes

    o, d = (torch.from_numpy(x).cuda() for x in scenes.incoherent_rays(400000, seed=3))
    mine, other = _scene(gpu_ctx, 60000), _scene(gpu_ctx, 50000, 2)
    tree = getattr(mine, kind)()
    want = [x.cpu().numpy() for x in tree.trace_closest(o, d, tri_eps=1e-12)]
    tree.close()
    stop, bad = threading.Event(), []

    def work():
        s = torch.cuda.Stream()
        try:
            while not stop.is_set():
                other.build_bvh_fast_device(s).close()
                other.build_bvh_device(s).close()
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    ts = [threading.Thread(target=work) for _ in range(3)]
    for t in ts:
        t.start()
    st = torch.cuda.Stream()
    outs = [(torch.empty(len(o), dtype=torch.int32, device="cuda"), torch.empty(len(o), device="cuda"))
            for _ in range(8)]
    torch.cuda.synchronize()
    for hit, t in outs:
        tree = getattr(mine, kind)(st)
        tree.trace_closest(o, d, hit, t, tri_eps=1e-12, stream=st)
        tree.close()
    stop.set()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    gpu_ctx.check()
    assert not bad
    for hit, t in outs:
        assert np.array_equal(hit.cpu().numpy(), want[0]) and np.array_equal(t.cpu().numpy(), want[1])
    mine.close()
    other.close()


def test_a_budget_of_zero_gives_back_what_is_kept(gpu_ctx):
    sc = _scene(gpu_ctx, 1000000)
    gpu_ctx.set_memory_budget(0)
    before = _free()
    sc.build_bvh_device().close()
    assert before - _free() > 128 << 20
    gpu_ctx.set_memory_budget(0)
    assert before - _free() < 64 << 20
    sc.close()


# Scratch of a build of 20,000 triangles when the nodes were held twice and a triangle
# record was 48 bytes: what a budget admitted then it still admits.
SCRATCH = {"build_bvh_device": 3214336, "build_bvh_fast_device": 6187520}


@pytest.mark.parametrize("kind", SCRATCH)
@pytest.mark.parametrize("scene", ["soup", "terrain"])
def test_a_budget_admits_what_it_did(gpu_ctx, kind, scene):
    from cudatracer_gb300 import api, scenes

    n = 20000
    s = scenes.soup_scene(n) if scene == "soup" else scenes.terrain_scene(grid=101, spheres=0)[0]
    sc = gpu_ctx.scene({"vertices": s.vertices, "normals": s.normals, "indices": s.indices[:n]}, [api.Material()])
    tree = getattr(sc, kind)()
    nodes, held = tree.info()["quad_node_count"], tree.info()["device_bytes"]
    tree.close()
    was = 2 * 128 * nodes + 48 * n + 4 * n
    assert held <= was
    gpu_ctx.set_memory_budget(gpu_ctx.device_bytes + SCRATCH[kind] + was)
    try:
        getattr(sc, kind)().close()
    finally:
        gpu_ctx.set_memory_budget(0)
    sc.close()
