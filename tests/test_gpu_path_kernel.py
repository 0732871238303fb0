"""Frames of few pixels run as one kernel (a path per thread). Its frames equal
the staged wavefront's bit for bit, ray counts included: the stages run when a
job is profiled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (33, 1), (5, 7), (32, 32), (67, 41), (362, 362), (363, 363)]  # 131,072 pixels is the largest


@pytest.fixture(scope="module")
def world(gpu_ctx):
    from cudatracer_gb300 import api, scenes

    ts, cam = scenes.material_zoo_scene(ground_textures=(32, 16))
    sc = gpu_ctx.scene(scenes.scene_arrays(ts), [api.Material(**m) for m in ts.materials], ts.textures,
                       ts.skybox_texture)
    return sc, sc.build_bvh(), sc.build_bvh_fast_device(), cam


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("mode", ["fast", "exact", "exact-shade", "fast full", "exact full", "no shadow"])
def test_path_kernel_equals_the_stages(gpu_ctx, world, size, mode):
    from cudatracer_gb300 import api

    sc, ref, fast, cam = world
    w, h = size
    math = {"fast": 0, "exact": 1}.get(mode.split()[0], 2)
    p = api.Params(w, h, camera=api.Camera(w, h, cam["fov"], cam["position"], cam["forward"], cam["up"]),
                   max_depth=1 if w == 33 else 6, exact_math=math, shading_mode=int("full" in mode),
                   shadow=mode != "no shadow", texture_filter=w % 2)
    got = []
    for staged in (False, True):
        job = api.RenderJob(gpu_ctx, w, h)
        job.profile(staged)
        p.reset(job)
        p.samples = 14
        job.stats(reset=True)
        api.launch_kernels(job, sc, ref if math == 1 else fast, p)
        gpu_ctx.check()
        got.append((job.accum_tensor().cpu().numpy().copy(), job.stats()))
        job.close()
    assert np.array_equal(got[0][0].view(np.int32), got[1][0].view(np.int32))
    assert got[0][1] == got[1][1]
    if w > 32:
        assert np.count_nonzero(got[0][0]) > 0
