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
    trees = [sc.build_bvh_fast_device() for _ in range(10)]
    held = sum(t.info()["device_bytes"] for t in trees)
    assert held > 3 * GIB // 2
    for t in trees:
        assert b.lib.ct_bvh_destroy(b.h, t.h) == 0
        t.h = None
    assert before - _free() <= GIB + (128 << 20)
    sc.close()
    b.close()
    a.close()
