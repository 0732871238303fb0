"""The device builders' subtrees of at most 16 primitives (built by one thread
each) at the edges of that range: the traversal-speed tree equals the host's
byte for byte, and the reference's tree its quad nodes and every leaf's
primitives, around 16 and 128 primitives (the sizes at which a range changes
hands), with centroid ties on one axis or all, and along chains whose subtrees
may and may not reach the depth limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(ctx, v, ix):
    from cudatracer_gb300 import api

    sc = ctx.scene({"vertices": v, "normals": np.ones_like(v), "indices": ix}, [api.Material()])
    h, d = sc.build_bvh_fast(), sc.build_bvh_fast_device()
    qh, ph = h.export()
    qd, pd = d.export()
    assert np.array_equal(ph, pd)
    assert np.array_equal(qh.view(np.int32), qd.view(np.int32))
    hr, dr = sc.build_bvh(), sc.build_bvh_device()
    qh, ph = hr.export()
    qd, pd = dr.export()
    assert np.array_equal(qh.view(np.int32), qd.view(np.int32))
    counts, childs = qh[:, 28:32], qh[:, 24:28]
    for first, cnt in zip(childs[counts > 0], counts[counts > 0]):
        assert np.array_equal(np.sort(ph[first:first + cnt]), np.sort(pd[first:first + cnt]))
    for x in (h, d, hr, dr, sc):
        x.close()


def _tris(c, rng, size=0.05):
    v = (c[:, None, :] + rng.normal(size=(c.shape[0], 3, 3)) * size).astype(np.float32)
    return v.reshape(-1, 3), np.arange(3 * c.shape[0], dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("ntri", [2, 3, 15, 16, 17, 31, 33, 127, 128, 129, 2000])
@pytest.mark.parametrize("ties", ["none", "one axis", "pairs", "all"])
def test_leaf_subtrees_equal_the_host(gpu_ctx, ntri, ties):
    rng = np.random.default_rng(ntri)
    c = rng.uniform(0, 1, size=(ntri, 3))
    if ties == "one axis":
        c[:, 1] = np.round(c[:, 1] * 3) / 3
    if ties == "all":
        c[:] = np.round(c * 2) / 2
    v, ix = _tris(c, rng) if ties in ("none", "one axis") else _tris(c, rng, 0.0)
    if ties in ("pairs", "all"):  # the same triangle about its centre: equal centroids stay equal
        shape = np.array([[0.02, 0, 0.01], [-0.02, 0.01, 0], [0, -0.01, -0.01]], np.float32)
        v = (v.reshape(-1, 3, 3) + shape[None]).reshape(-1, 3).astype(np.float32)
    if ties == "pairs":
        v.reshape(-1, 9)[1::2] = v.reshape(-1, 9)[0::2][: v.shape[0] // 3 // 2]
    _compare(gpu_ctx, v, ix)


@pytest.mark.parametrize("ntri", [58, 60, 61, 62, 63, 70, 76, 80])
@pytest.mark.parametrize("step", [2.0, 1.5, 32.0])
def test_chains_around_the_depth_limit(gpu_ctx, ntri, step):
    xs = (np.float64(step) ** -np.arange(ntri) * 1e3).astype(np.float32)
    v = np.zeros((3 * ntri, 3), np.float32)
    v[:, 0] = np.repeat(xs, 3)
    v[1::3, 1] = xs
    v[2::3, 2] = xs
    _compare(gpu_ctx, v, np.arange(3 * ntri, dtype=np.uint32).reshape(-1, 3))
