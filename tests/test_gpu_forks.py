"""A pass's connect runs beside the next pass's extend, in a batch's graph and in large
iterations of the server. The last pass follows at once where depths are 1 and 2, jobs of
different depths share the queues, and results are those of one stage after another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEPTHS = [(1,), (2,), (3,), (1, 2), (2, 1, 5)]


@pytest.fixture(scope="module")
def world(gpu_ctx):
    from cudatracer_gb300 import api, scenes

    ts, cam = scenes.terrain_scene(grid=64, spheres=8, seed=9, extent=60.0, sky_size=(128, 64))
    sc = gpu_ctx.scene(scenes.scene_arrays(ts), [api.Material(**m) for m in ts.materials], ts.textures,
                       ts.skybox_texture)
    return sc, sc.build_bvh_device(), dict(cam, position=(0.0, 14.0, 34.0))


def _jobs(world, depths, w, h, spp):
    from cudatracer_gb300 import api

    sc, tree, cam = world
    out = []
    for k, d in enumerate(depths):
        p = api.default_params(w + 7 * k, h + 3 * k)
        p.max_depth, p.frame_index = d, 2 * k
        out.append(dict(scene=sc, bvh=tree, params=p, spp=spp + k,
                        camera=api.Camera(p.width, p.height, cam["fov"], cam["position"], cam["forward"], cam["up"])))
    return out


def _batch(gpu_ctx, jobs, math, **tuning):
    import torch

    from cudatracer_gb300 import api

    b = api.Batch(gpu_ctx, jobs, exact_math=math)
    b.set_tuning(extend_block=128, connect_block=128, shade_waves=1, **tuning)
    b.run()
    torch.cuda.synchronize()
    gpu_ctx.check()
    out, st = [b.accum_tensor(k).cpu().numpy().copy() for k in range(len(jobs))], b.stats()
    b.close()
    return out, st


@pytest.mark.parametrize("depths", DEPTHS)
@pytest.mark.parametrize("math", [0, 1, 2])
def test_batch_graph_equals_the_chain(gpu_ctx, world, depths, math):
    jobs = _jobs(world, depths, 61, 47, 5)
    want, ws = _batch(gpu_ctx, jobs, math, use_graph=0)
    for sort in (0, 1):
        got, gs = _batch(gpu_ctx, jobs, math, use_graph=1, sort_key=sort)
        assert gs == ws
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.int32), b.view(np.int32))
    if max(depths) > 1:
        assert ws["shadow_rays"] > 0


# 257x256 and up: over 65,536 pixel-samples an iteration, so each connect but the last is forked
@pytest.mark.parametrize("depths", DEPTHS)
@pytest.mark.parametrize("math", [0, 1, 2])
def test_served_results_do_not_depend_on_the_fork(gpu_ctx, world, depths, math):
    from cudatracer_gb300 import api

    jobs = _jobs(world, depths, 257, 256, 3)
    srv = api.Server(gpu_ctx, max_inflight_pixels=1 << 20, iter_pixels=1, exact_math=math)  # a sample a job at a time
    alone = [srv.wait(srv.submit_render(j))[1] for j in jobs]
    ids = [srv.submit_render(j) for j in jobs]
    mixed = [srv.wait(i)[1] for i in ids]
    srv.close()
    gpu_ctx.check()
    want, _ = _batch(gpu_ctx, jobs, math, use_graph=0)
    for j, a, m, w in zip(jobs, alone, mixed, want):
        assert np.array_equal(a.view(np.int32), m.view(np.int32))
        assert np.allclose(a, w.reshape(a.shape), rtol=1e-5, atol=1e-6)
        if math == 1:
            assert np.array_equal(a.view(np.int32), _two_slots(gpu_ctx, j).reshape(a.shape).view(np.int32))


def _two_slots(gpu_ctx, j):
    """The server's summation of bit-exact samples: sample i in slot i mod 2, the slots added in order."""
    from cudatracer_gb300 import api

    total = None
    for slot in range(min(j["spp"], 2)):
        job = api.RenderJob(gpu_ctx, j["params"].width, j["params"].height)
        job.reset()
        for i in range(slot, j["spp"], 2):
            p = api.default_params(j["params"].width, j["params"].height)
            p.max_depth, p.exact_math = j["params"].max_depth, 1
            p.frame_index = j["params"].frame_index + 2 * i
            job.accumulate(j["scene"], j["bvh"], j["camera"], p)
        gpu_ctx.check()
        got = job.accum_tensor().cpu().numpy().copy()
        job.close()
        total = got if total is None else total + got
    return total
