"""Frames of more than 131,072 pixels run as wavefront stages, several frames in flight:
more frames than slots, logs that grow, sorted bounce queues. Odd size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 385, 347
SLOTS = 10


@pytest.fixture(scope="module")
def world(gpu_ctx):
    from cudatracer_gb300 import api, scenes

    ts, cam = scenes.terrain_scene(grid=96, spheres=10, seed=5, extent=60.0, sky_size=(128, 64))
    sc = gpu_ctx.scene(scenes.scene_arrays(ts), [api.Material(**m) for m in ts.materials], ts.textures,
                       ts.skybox_texture)
    cam = dict(cam, position=(0.0, 14.0, 34.0))
    return sc, sc.build_bvh_device(), sc.build_bvh_fast_device(), cam


def _frames(gpu_ctx, world, math, depths, first=0, profiled=False, ray_sort=0):
    import torch

    from cudatracer_gb300 import api

    sc, ref, fast, cam = world
    job = api.RenderJob(gpu_ctx, W, H)
    job.profile(profiled)
    p = api.Params(W, H, camera=api.Camera(W, H, cam["fov"], cam["position"], cam["forward"], cam["up"]),
                   exact_math=math, ray_sort=ray_sort)
    p.reset(job)
    p.samples = 2 * first
    for d in depths:
        p.max_depth = d
        api.launch_kernels(job, sc, ref if math == 1 else fast, p)
    torch.cuda.synchronize()
    gpu_ctx.check()
    out = job.accum_tensor().cpu().numpy().copy()
    job.close()
    return out


def _same(a, b):
    return np.array_equal(a.view(np.int32), b.view(np.int32))


@pytest.mark.parametrize("math", [0, 2])
def test_frames_in_flight_equal_frames_one_by_one(gpu_ctx, world, math):
    """Each frame rendered by a job of its own, added up in frame order as the fold does."""
    depths = [3 + k % 4 for k in range(2 * SLOTS + 3)]
    want = np.zeros((W * H, 4), np.float32)
    for k, d in enumerate(depths):
        want = want + _frames(gpu_ctx, world, math, [d], first=k)
    got = _frames(gpu_ctx, world, math, depths)
    assert _same(got, want) and got[:, 3].sum() > 0


def test_exact_frames_in_flight_equal_frames_in_sequence(gpu_ctx, world):
    """Logs are reused (six slots) and grow with the depth; profiling runs frames in sequence."""
    depths = [4] * 15 + [9] * 8
    assert _same(_frames(gpu_ctx, world, 1, depths), _frames(gpu_ctx, world, 1, depths, profiled=True))


@pytest.mark.parametrize("math", [0, 1, 2])
@pytest.mark.parametrize("profiled", [False, True])
def test_ray_sort_keys_change_no_frame(gpu_ctx, world, math, profiled):
    from cudatracer_gb300 import _lib

    outs = [_frames(gpu_ctx, world, math, [6, 5, 6], profiled=profiled, ray_sort=k)
            for k in (_lib.CT_SORT_NONE, _lib.CT_SORT_OCTANT, _lib.CT_SORT_FACE_CELLS)]
    assert _same(outs[0], outs[1]) and _same(outs[0], outs[2]) and outs[0][:, 3].sum() > 0
