"""The device builders' level kernels (nodes of more than 128 primitives) at the
edges of chunks and of levels issued together: nodes that are halved as they lie or
stay leaves because their centroids coincide, unbalanced trees with a large node on
many levels, and sizes around the chunks' and the warps' limits. Compared with the
host's trees as the leaf subtrees are (byte for byte; the reference's leaves as
sets)."""
import numpy as np
import pytest

from tests.test_gpu_bvh_leaf_tasks import _compare

pytestmark = pytest.mark.gpu


def _scene(centres, rng, size):
    shape = rng.normal(size=(3, 3)) * size if np.isscalar(size) else size
    v = (centres[:, None, :] + shape).astype(np.float32).reshape(-1, 3)
    return v, np.arange(v.shape[0], dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("ntri", [129, 255, 256, 257, 511, 513, 2047, 2049, 20480, 33000])
@pytest.mark.parametrize("kind", ["uniform", "coincident", "clusters", "chain", "line"])
def test_level_kernels_equal_the_host(gpu_ctx, ntri, kind):
    rng = np.random.default_rng(ntri)
    c = rng.uniform(-1, 1, size=(ntri, 3))
    size = 0.02
    if kind == "coincident":  # one place, but for a few
        c[:] = 0.25
        c[: ntri // 100] = rng.uniform(-1, 1, size=(ntri // 100, 3))
    if kind == "clusters":  # a few places, of very different population, in random order
        place = rng.uniform(-1, 1, size=(6, 3))
        c = place[rng.choice(6, ntri, p=[0.6, 0.2, 0.1, 0.05, 0.03, 0.02])]
    if kind == "chain":  # halving distances: one large node a level
        c *= 2.0 ** -(np.arange(ntri) // max(1, ntri // 40))[:, None]
        size = 1e-4
    if kind == "line":
        c[:, 1:] = 0.0
    v, ix = _scene(c, rng, size)
    _compare(gpu_ctx, v, ix)


@pytest.mark.parametrize("ntri", [100001, 1000001])
def test_mid_size_rules_equal_the_host(gpu_ctx, ntri):
    """Past the sizes at which the blocks for mid-size nodes change (256 threads, 1,024 primitives)."""
    rng = np.random.default_rng(ntri)
    v, ix = _scene(rng.uniform(-1, 1, size=(ntri, 3)), rng, 0.004)
    _compare(gpu_ctx, v, ix)
