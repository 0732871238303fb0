"""Small queries and frames, whose rays are spread over more warps with fewer
lanes at work each, give what the same rays give in a call of full warps."""
import numpy as np
import pytest

from tests import test_gpu_path_kernel as path_kernel

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 767, 768, 769, 1537, 5000, 31 * 768, 31 * 768 + 1, 32 * 768 + 1)


@pytest.mark.parametrize("kind", ["build_bvh", "build_bvh_fast_device", "build_bvh_wide"])
def test_small_queries_equal_a_large_one(gpu_ctx, kind):
    import torch

    from cudatracer_gb300 import api, scenes

    s = scenes.soup_scene(30000, seed=5)
    sc = gpu_ctx.scene({"vertices": s.vertices, "normals": s.normals, "indices": s.indices}, [api.Material()])
    b = getattr(sc, kind)()
    o, d = (torch.from_numpy(x).cuda() for x in scenes.incoherent_rays(70000, seed=6))
    h, t = b.trace_closest(o, d, tri_eps=1e-12)
    occ = b.trace_any(o, d, tri_eps=1e-12)
    assert (h >= 0).sum() > 1000 and occ.sum() > 1000
    for n in SIZES:
        hn, tn = b.trace_closest(o[:n].contiguous(), d[:n].contiguous(), tri_eps=1e-12)
        on = b.trace_any(o[:n].contiguous(), d[:n].contiguous(), tri_eps=1e-12)
        gpu_ctx.check()
        assert torch.equal(hn, h[:n]) and torch.equal(on, occ[:n]), n
        assert np.array_equal(tn.cpu().numpy().view(np.int32), t[:n].cpu().numpy().view(np.int32)), n


world = path_kernel.world


@pytest.mark.parametrize("size", [(48, 16), (769, 1), (64, 48), (154, 154), (155, 155)])
@pytest.mark.parametrize("mode", ["fast", "exact", "exact-shade full"])
def test_small_frames_equal_the_stages(gpu_ctx, world, size, mode):
    path_kernel.test_path_kernel_equals_the_stages(gpu_ctx, world, size, mode)
