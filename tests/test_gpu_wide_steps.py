"""The wide-tree query kernel's steps: nodes of every fill, more pending entries
than the shared part of the stack holds, and plane offsets that overflow.

Closest hits (ids equal, t within the documented 1e-5 relative) and occlusion
equal the FP64 oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind, ntri):
    rng = np.random.default_rng(ntri)
    if kind == "crossing":  # every triangle reaches across the middle: all boxes overlap, stacks grow deep
        a = rng.normal(size=(ntri, 3))
        b = rng.normal(size=(ntri, 3))
        c = rng.uniform(-0.05, 0.05, (ntri, 3))
        tri = np.stack([a + c, b + c, c - a - b], axis=1) + 0.5
    else:
        tri = rng.uniform(0, 1, (ntri, 1, 3)) + rng.normal(size=(ntri, 3, 3)) * 0.05
    v = np.ascontiguousarray(tri.reshape(-1, 3), np.float32)
    return v, np.arange(3 * ntri, dtype=np.uint32).reshape(-1, 3)


def _rays(n, axis):
    rng = np.random.default_rng(n)
    o = np.zeros((n, 4), np.float32)
    d = np.zeros((n, 4), np.float32)
    o[:, :3] = rng.uniform(-1, 2, (n, 3))
    if axis:
        d[np.arange(n), np.arange(n) % 3] = np.where(np.arange(n) % 2, 1.0, -1.0)
    else:
        e = 0.5 + rng.normal(size=(n, 3)) * 0.1 - o[:, :3]
        d[:, :3] = e / np.linalg.norm(e, axis=1, keepdims=True)
    d[:, 3] = 1e34
    return o, d


def _fp64(orc, v, ix, ob, o, d, any_hit=False):
    """The oracle; the reference's tree of one or two triangles is empty, so there each triangle in turn."""
    if len(ix) > 2:
        return orc.trace_fp64(v, ix, ob["quad"], ob["prims"], o, d, any_hit=any_hit)
    h, t = np.full(len(o), -1, np.int32), d[:, 3].astype(np.float64)
    org, dr = o[:, :3].astype(np.float64), d[:, :3].astype(np.float64)
    for k, (a, b, c) in enumerate(v[ix].astype(np.float64)):
        p = np.cross(dr, c - a)
        q = np.cross(org - a, b - a)
        with np.errstate(divide="ignore", invalid="ignore"):
            inv = 1.0 / (p @ (b - a))
            u, w, s = ((org - a) * p).sum(1) * inv, (dr * q).sum(1) * inv, (q @ (c - a)) * inv
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (s > 0) & (s < t)
        h[ok], t[ok] = k, s[ok]
    return h, t


@pytest.mark.parametrize(
    "kind,ntri,n,axis,scale",
    [("soup", k, 257, False, 1.0) for k in (1, 2, 7, 8, 9, 25, 70)]
    + [("soup", 3000, n, False, 1.0) for n in (1, 31, 33, 20001)]
    + [("crossing", 400, 3000, False, 1.0), ("crossing", 6000, 3000, False, 1.0)]
    # an axis-parallel ray's offset overflows from node steps of 1e4 on (extents of 2.6e6)
    + [("soup", 3000, 3000, True, 2.0**20), ("soup", 3000, 3000, True, 2.0**32), ("crossing", 400, 3000, True, 2.0**32)],
)
def test_wide_steps_equal_fp64(gpu_ctx, orc, kind, ntri, n, axis, scale):
    import torch

    from cudatracer_gb300 import api

    v, ix = _scene(kind, ntri)
    o, d = _rays(n, axis)
    # a power of two scales positions, and t, exactly: the oracle's answer is the unit scene's
    ob = orc.bvh_build(v, ix)
    ho, to = _fp64(orc, v, ix, ob, o, d)
    arr = {"vertices": v * np.float32(scale), "normals": np.tile(np.array([[0, 0, 1]], np.float32), (v.shape[0], 1)),
           "indices": ix}
    wb = gpu_ctx.scene(arr, [api.Material()]).build_bvh_wide()
    od = o.copy()
    od[:, :3] *= np.float32(scale)
    O = torch.from_numpy(od).cuda()
    h, t = wb.trace_closest(O, torch.from_numpy(d).cuda())
    gpu_ctx.check()
    h, t = h.cpu().numpy(), t.cpu().numpy()
    assert np.array_equal(h, ho)
    hit = ho >= 0
    assert (np.abs(t[hit].astype(np.float64) / scale - to[hit]) <= 1e-5 * to[hit]).all()
    # finite ranges around the hit
    d2 = d.copy()
    near = np.where(hit, to, 1.0) * np.where(np.arange(n) % 2, 1.001, 0.999)
    d2[:, 3] = near
    occ, _ = _fp64(orc, v, ix, ob, o, d2, any_hit=True)
    d3 = d2.copy()
    d3[:, 3] = d2[:, 3] * np.float32(scale)
    got = wb.trace_any(O, torch.from_numpy(d3).cuda())
    gpu_ctx.check()
    assert np.array_equal(got.cpu().numpy().astype(bool), occ >= 0)


def test_export_of_several_pieces(gpu_ctx):
    """More than 65,536 nodes: the device's form goes back to the 80-byte one in pieces."""
    from cudatracer_gb300 import _lib, scenes
    from tests.test_gpu_wide import _check_structure
    from tests.test_gpu_wide import _scene as scene_of

    s = scenes.soup_scene(300000, seed=77)
    b = scene_of(gpu_ctx, s.vertices, s.indices).build_bvh_wide()
    nodes, prims = b.export(_lib.CT_BVH_WIDE8_Q8)
    assert nodes.shape[0] > 65536
    _check_structure(s.vertices, s.indices, nodes, prims)
