"""Where frames go from one kernel to the stages: 81,920 pixels, with the reference's
traversal 131,072. Both sides of the line give the profiled stages' bits, and a frame on
the one-kernel side is no slower than a larger one on the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(gpu_ctx):
    from cudatracer_gb300 import api, scenes

    ts, cam = scenes.material_zoo_scene(ground_textures=(32, 16))
    sc = gpu_ctx.scene(scenes.scene_arrays(ts), [api.Material(**m) for m in ts.materials], ts.textures,
                       ts.skybox_texture)
    return sc, sc.build_bvh(), sc.build_bvh_fast_device(), cam


def _params(w, h, cam, mode):
    from cudatracer_gb300 import api

    math = {"fast": 0, "exact": 1}.get(mode.split()[0], 2)
    return api.Params(w, h, camera=api.Camera(w, h, cam["fov"], cam["position"], cam["forward"], cam["up"]),
                      max_depth=5, exact_math=math, shading_mode=int("full" in mode))


@pytest.mark.parametrize("size", [(4096, 20), (241, 340), (4097, 20), (512, 256), (513, 256)])
@pytest.mark.parametrize("mode", ["fast", "exact", "exact-shade", "fast full", "exact full"])
def test_both_sides_equal_the_stages(gpu_ctx, world, size, mode):
    from cudatracer_gb300 import api

    sc, ref, fast, cam = world
    w, h = size
    p = _params(w, h, cam, mode)
    got = []
    for staged in (False, True):
        job = api.RenderJob(gpu_ctx, w, h)
        job.profile(staged)
        p.reset(job)
        p.samples = 6
        job.stats(reset=True)
        api.launch_kernels(job, sc, ref if mode.startswith("exact") and "-" not in mode else fast, p)
        gpu_ctx.check()
        got.append((job.accum_tensor().cpu().numpy().copy(), job.stats()))
        job.close()
    assert np.array_equal(got[0][0].view(np.int32), got[1][0].view(np.int32))
    assert got[0][1] == got[1][1]
    assert np.count_nonzero(got[0][0]) > 0


def _frames_ms(gpu_ctx, world, side, mode):
    import torch

    from cudatracer_gb300 import api

    sc, _, fast, cam = world
    p = _params(side, side, cam, mode)
    job = api.RenderJob(gpu_ctx, side, side)
    best = float("inf")
    for _ in range(12):
        p.reset(job)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(16):
            api.launch_kernels(job, sc, fast, p)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    job.close()
    return best


# 400x400 runs the stages and has 22 % more pixels
@pytest.mark.parametrize("mode", ["fast", "exact-shade full"])
def test_fewer_pixels_take_no_longer(gpu_ctx, world, mode):
    small, large = _frames_ms(gpu_ctx, world, 362, mode), _frames_ms(gpu_ctx, world, 400, mode)
    assert small <= large, (small, large)
