"""Memory of device builds: kept between builds inside the context, counted
while a tree holds it, refused over the budget, and safe with several threads
and streams building, tracing and destroying at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ("build_bvh_device", "build_bvh_fast_device", "build_bvh_wide")


def _scene(ctx, n, seed):
    from cudatracer_gb300 import api, scenes

    s = scenes.soup_scene(n, seed=seed)
    return ctx.scene({"vertices": s.vertices, "normals": s.normals, "indices": s.indices}, [api.Material()])


@pytest.mark.parametrize("kind", KINDS)
def test_bytes_are_counted_and_given_back(gpu_ctx, kind):
    from cudatracer_gb300 import _lib

    sc = _scene(gpu_ctx, 3000, 1)
    used = gpu_ctx.device_bytes
    b = getattr(sc, kind)()
    held = gpu_ctx.device_bytes - used
    assert held == b.info()["device_bytes"] and held > 3000 * 48
    b.close()
    assert gpu_ctx.device_bytes == used
    gpu_ctx.set_memory_budget(used + held // 2)
    try:
        with pytest.raises(_lib.CTError) as e:
            getattr(sc, kind)()
        assert e.value.status == 2 and gpu_ctx.device_bytes == used
    finally:
        gpu_ctx.set_memory_budget(0)
    getattr(sc, kind)().close()
    sc.close()


def test_threads_build_trace_and_destroy_at_once(gpu_ctx):
    import torch

    from cudatracer_gb300 import scenes

    o, d = (torch.from_numpy(x).cuda() for x in scenes.incoherent_rays(20000, seed=3))
    sizes = (150, 2500, 40000)
    want, scs = {}, {}
    for n in sizes:
        scs[n] = _scene(gpu_ctx, n, n)
        for kind in KINDS:
            b = getattr(scs[n], kind)()
            want[n, kind] = [x.cpu().numpy() for x in b.trace_any(o, d, tri_eps=1e-12).view(1, -1)]
            b.close()
    bad = []

    def work(k):
        st = torch.cuda.Stream()
        try:
            for i in range(6):
                n, kind = sizes[(k + i) % 3], KINDS[(k + 2 * i) % 3]
                if kind == "build_bvh_wide":  # its queries share the context's record buffer
                    getattr(scs[n], kind)(st).close()
                    continue
                b = getattr(scs[n], kind)(st)
                q, _ = b.export()
                r = getattr(scs[n], kind)(st)
                if not np.array_equal(q.view(np.int32), r.export()[0].view(np.int32)):
                    bad.append((k, i, "trees differ"))
                r.close()
                b.close()
        except Exception as e:  # noqa: BLE001
            bad.append((k, repr(e)))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for n in sizes:
        for kind in KINDS:
            b = getattr(scs[n], kind)()
            got = [x.cpu().numpy() for x in b.trace_any(o, d, tri_eps=1e-12).view(1, -1)]
            assert np.array_equal(got, want[n, kind])
            b.close()
        scs[n].close()
    gpu_ctx.check()
