"""The ray step of the quad traversal (two triangles or one node per step, exact
slabs in hardware min/max): closest and any hits equal the oracle's bit for bit
where the step can go wrong. Every triangle is there twice, so the winner of an
exact t tie shows the order in which nodes and triangles were visited."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(ntri, seed):
    rng = np.random.default_rng(seed)
    half = (ntri + 1) // 2
    c = rng.uniform(0.0, 1.0, size=(half, 1, 3))
    v = (c + rng.normal(size=(half, 3, 3)) * 0.15).astype(np.float32)
    v = np.concatenate([v, v])[:ntri]  # coincident pairs (one unpaired when ntri is odd)
    return v.reshape(-1, 3), np.arange(3 * ntri, dtype=np.uint32).reshape(-1, 3)


def _rays(quad, n, seed):
    """Random rays; rays from the corners of node boxes (origins on two or three planes at once), towards every
    octant, along the axes and within the planes."""
    rng = np.random.default_rng(seed)
    o = rng.uniform(-0.2, 1.2, size=(n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    f = quad.view(np.float32).reshape(-1, 32)[:, :24].reshape(-1, 3, 2, 4)  # node, axis, min/max, child
    k = n * 3 // 4
    node, child = rng.integers(0, f.shape[0], k), rng.integers(0, 4, k)
    for a in range(3):
        p = f[node, a, rng.integers(0, 2, k), child]
        keep = np.isfinite(p) & (np.abs(p) < 1e30) & (rng.uniform(size=k) < 0.8)
        o[:k, a] = np.where(keep, p, o[:k, a])
    zero = rng.uniform(size=(n, 3)) < 0.15
    zero[zero.all(1)] = False
    d[zero] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o, d.astype(np.float32)


def _t4(a, w):
    import torch

    return torch.from_numpy(np.concatenate([a, np.broadcast_to(np.asarray(w, np.float32), (a.shape[0],))[:, None]],
                                           1).astype(np.float32)).cuda()


def _check(ctx, orc, bvh, quad, prims, v, ix, seed):
    o, d = _rays(quad, 6000, seed)
    hit, t = bvh.trace_closest(_t4(o, 0), _t4(d, 1e34), tri_eps=1e-7)
    oh, ot = orc.trace_closest(quad, prims, v, ix, o, d, eps=1e-7)
    ctx.check()
    assert np.array_equal(hit.cpu().numpy(), oh)
    assert np.array_equal(t.cpu().numpy().view(np.int32), ot.view(np.int32))
    tmax = np.where(ot < 1e30, ot * np.float32(1.25), np.float32(0.5)).astype(np.float32)
    tmax[::2] *= np.float32(0.5)
    occ = bvh.trace_any(_t4(o, 0), _t4(d, tmax), tri_eps=1e-7)
    ctx.check()
    assert np.array_equal(occ.cpu().numpy(), orc.trace_any(quad, prims, v, ix, o, d, tmax, eps=1e-7))


@pytest.mark.parametrize("ntri", [1, 2, 3, 4, 5, 31, 700])
@pytest.mark.parametrize("tree", ["reference", "fast"])
def test_ray_steps_equal_the_oracle(gpu_ctx, orc, tree, ntri):
    from cudatracer_gb300 import _lib, api

    v, ix = _soup(ntri, ntri)
    sc = gpu_ctx.scene({"vertices": v, "normals": np.ones_like(v), "indices": ix}, [api.Material()])
    for bvh in ((sc.build_bvh(), sc.build_bvh_device()) if tree == "reference" else
                (sc.build_bvh_fast(), sc.build_bvh_fast_device())):
        quad, prims = bvh.export(_lib.CT_BVH_QUAD)
        _check(gpu_ctx, orc, bvh, quad, prims, v, ix, 17 + ntri)
        bvh.close()
    sc.close()


@pytest.mark.parametrize("plane", [np.inf, np.nan, 3.4e38])
def test_imported_trees_with_planes_out_of_range(gpu_ctx, orc, plane):
    """Imported nodes may hold any plane: infinite, NaN, or so large that a slab term overflows."""
    from cudatracer_gb300 import api

    v, ix = _soup(300, 9)
    sc = gpu_ctx.scene({"vertices": v, "normals": np.ones_like(v), "indices": ix}, [api.Material()])
    b = orc.bvh_build(v, ix)
    quad = b["quad"].copy()
    f = quad.view(np.float32)
    rng = np.random.default_rng(3)
    rows = rng.integers(0, f.shape[0], 40)
    f[rows, rng.choice([4, 5, 12, 13, 20, 21], 40)] = plane  # max planes of children 0 and 1
    f[rows[:20], rng.choice([0, 8, 16], 20)] = -plane
    bvh = sc.import_quad(quad, b["prims"])
    _check(gpu_ctx, orc, bvh, quad, b["prims"], v, ix, 4)
    bvh.close()
    sc.close()
