"""What a wide-tree query costs whatever its rays do: rays that miss the scene's box
read one node each, so the launches are all there is.

A wide query is a counter fill, the traversal and the settlement of its records; a
quad query is the first two. Hence the bound: the quad query of the same rays, half as
much again for the larger root node and the ray set-up, and 6 us for one launch more."""
import pytest

pytestmark = pytest.mark.gpu


def _best_us(call):
    import torch

    best = float("inf")
    for k in range(80):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(4):
            call()
        b.record()
        torch.cuda.synchronize()
        if k >= 20:
            best = min(best, a.elapsed_time(b) * 1000.0 / 4)
    return best


@pytest.fixture(scope="module")
def trees(gpu_ctx):
    from cudatracer_gb300 import api, scenes

    s = scenes.sphere_scene(3)
    sc = gpu_ctx.scene(scenes.scene_arrays(s), [api.Material(**m) for m in s.materials], s.textures, s.skybox_texture)
    yield sc.build_bvh_wide(), sc.build_bvh_fast_device()


def _cost(trees, n, any_hit):
    import torch

    wide, quad = trees
    o = torch.zeros(n, 4, device="cuda")
    o[:, 2] = 5.0
    d = torch.zeros(n, 4, device="cuda")
    d[:, 2] = 1.0  # away from the unit sphere
    d[:, 3] = 10.0
    occ = torch.empty(n, dtype=torch.uint8, device="cuda")
    hit, t = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda")
    if any_hit:
        return tuple(_best_us(lambda: x.trace_any(o, d, occ)) for x in (wide, quad))
    return tuple(_best_us(lambda: x.trace_closest(o, d, hit, t)) for x in (wide, quad))


# 4,096: rays spread over 768 warps; 155,648: every lane of the chip has one
@pytest.mark.parametrize("n", [64, 4096, 155648])
@pytest.mark.parametrize("any_hit", [False, True])
def test_rays_that_miss_cost_the_launches(trees, n, any_hit):
    wide, quad = _cost(trees, n, any_hit)
    assert wide <= 1.5 * quad + 6.0, (wide, quad)


@pytest.mark.parametrize("n", [1, 33, 4096, 24577, 100001])
def test_query_counters_count_every_ray_once(trees, n):
    import torch

    wide = trees[0]
    g = torch.Generator(device="cuda").manual_seed(n)
    o = torch.zeros(n, 4, device="cuda")
    o[:, :3] = torch.rand(n, 3, generator=g, device="cuda") * 4.0 - 2.0
    d = torch.zeros(n, 4, device="cuda")
    d[:, :3] = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
    d[:, 3] = 1e34
    wide.wide_stats(reset=True)
    wide.trace_closest(o, d)
    wide.trace_any(o, d)
    torch.cuda.synchronize()
    assert wide.wide_stats(reset=True)["rays"] == 2 * n
