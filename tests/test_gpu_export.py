"""Exports of device-built trees: at the size of a piece, with no memory to be had, under
capture, and not slower than a few copies of the bytes."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PIECE = 1 << 19  # nodes converted at a time
KINDS = ("build_bvh_device", "build_bvh_fast_device", "build_bvh_wide")


def _scene(ctx, n):
    from cudatracer_gb300 import api, scenes

    s = scenes.soup_scene(n, seed=3)
    return ctx.scene({"vertices": s.vertices, "normals": s.normals, "indices": s.indices}, [api.Material()])


def _export(b, kind, offset=0):
    """The nodes, into a buffer that starts `offset` bytes off an aligned one."""
    from cudatracer_gb300 import _lib

    wide = kind == "build_bvh_wide"
    nbytes = b.info()["quad_node_count"] * (80 if wide else 128)
    buf = np.full(nbytes + 64, 0xA5, np.uint8)
    at = buf.ctypes.data + offset
    st = b.ctx.lib.ct_bvh_export(b.h, _lib.CT_BVH_WIDE8_Q8 if wide else _lib.CT_BVH_QUAD, ctypes.c_void_p(at), None)
    assert st == 0
    assert (buf[:offset] == 0xA5).all() and (buf[offset + nbytes :] == 0xA5).all()
    return buf[offset : offset + nbytes].copy()


def _leaf_prims(nodes):
    """Every child of a quad export is named once, leaves are disjoint and cover the list."""
    q = nodes.view(np.int32).reshape(-1, 32)
    childs, counts = q[:, 24:28], q[:, 28:32]
    inner = childs[(counts == -1)]
    assert np.array_equal(np.sort(inner), np.arange(1, len(q)))
    leaf = counts > 0
    first, cnt = childs[leaf].astype(np.int64), counts[leaf].astype(np.int64)
    o = np.argsort(first)
    assert first[o][0] == 0 and np.array_equal(first[o][1:], (first + cnt)[o][:-1])
    assert (childs[counts == 0] == -1).all()
    return int(cnt.sum())


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 9, 3000, 1400000])
def test_pieces_and_offsets(gpu_ctx, kind, n):
    sc = _scene(gpu_ctx, n)
    b = getattr(sc, kind)()
    a = _export(b, kind)
    if n == 1400000 and kind == "build_bvh_fast_device":
        assert len(a) > PIECE * 128
    for offset in (1, 7, 16):
        assert np.array_equal(_export(b, kind, offset), a)
    if kind != "build_bvh_wide":
        assert _leaf_prims(a) == n
    b.close()
    sc.close()


@pytest.mark.parametrize("kind", KINDS)
def test_with_no_device_memory_left(gpu_ctx, kind):
    import torch

    sc = _scene(gpu_ctx, 400000)
    b = getattr(sc, kind)()
    want = _export(b, kind)
    hold, step = [], 16 << 30
    torch.cuda.synchronize()
    try:
        while step >= 1 << 21:
            try:
                hold.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                step //= 2
        assert np.array_equal(_export(b, kind, 1), want)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    b.close()
    sc.close()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("mode", ["global", "relaxed"])
def test_while_a_graph_is_captured(gpu_ctx, kind, mode):
    import torch

    sc = _scene(gpu_ctx, 3000)
    b = getattr(sc, kind)()
    want = _export(b, kind)
    x = torch.zeros(64, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        x += 1
        got = _export(b, kind)
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert x[0].item() == 2
    assert np.array_equal(got, want)
    b.close()
    sc.close()


def test_a_budget_gets_the_memory_back(lib):
    from cudatracer_gb300 import api

    ctx = api.Context(0)
    sc = _scene(ctx, 400000)
    b = sc.build_bvh_fast_device()
    used = ctx.device_bytes
    want = _export(b, "build_bvh_fast_device")
    ctx.set_memory_budget(used)  # nothing left in it
    assert np.array_equal(_export(b, "build_bvh_fast_device"), want)
    assert ctx.device_bytes == used
    b.close()
    sc.close()
    ctx.close()


@pytest.mark.parametrize("kind", KINDS)
def test_cost_of_an_export(gpu_ctx, kind):
    """2 M triangles: at most four plain copies of the bytes and half a millisecond."""
    import torch

    from cudatracer_gb300 import _lib

    sc = _scene(gpu_ctx, 2000000)
    b = getattr(sc, kind)()
    wide = kind == "build_bvh_wide"
    nbytes = b.info()["quad_node_count"] * (80 if wide else 128)
    dev, host = torch.zeros(nbytes, dtype=torch.uint8, device="cuda"), torch.zeros(nbytes, dtype=torch.uint8)
    lay = _lib.CT_BVH_WIDE8_Q8 if wide else _lib.CT_BVH_QUAD
    copy, export = [], []
    for _ in range(8):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        host.copy_(dev)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        assert b.ctx.lib.ct_bvh_export(b.h, lay, ctypes.c_void_p(host.data_ptr()), None) == 0
        copy.append(t1 - t0)
        export.append(time.perf_counter() - t1)
    b.close()
    sc.close()
    print(kind, nbytes, min(copy) * 1e3, min(export) * 1e3)
    assert min(export) <= 4 * min(copy) + 0.5e-3, (min(export), min(copy))
