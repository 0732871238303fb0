"""Both sides of the sizes at which the device builders change the blocks for mid-size
nodes (512 to 256 threads above 250,000 triangles, 2,048 to 1,024 primitives above
400,000): the trees are the host's."""
import numpy as np
import pytest

from tests.test_gpu_bvh_leaf_tasks import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntri", [250000, 250001, 400000, 400001])
def test_both_sides_equal_the_host(gpu_ctx, ntri):
    rng = np.random.default_rng(ntri)
    v = (rng.uniform(-1, 1, size=(ntri, 1, 3)) + rng.normal(size=(3, 3)) * 0.006).astype(np.float32).reshape(-1, 3)
    _compare(gpu_ctx, v, np.arange(3 * ntri, dtype=np.uint32).reshape(-1, 3))
