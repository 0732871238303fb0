"""Batch stages spread few rays over more warps, fewer lanes at work each; a job's
accumulation stays the same bits where a warp has one, some and all of its lanes
(1,024 rays a lane), alone and beside a job that fills the warps."""
import numpy as np
import pytest

from tests.test_gpu_batch import _job, _run, scenes_  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (33, 31), (32, 32), (41, 25), (181, 181), (182, 181)])
@pytest.mark.parametrize("exact", [0, 1, 2])
def test_batch_lanes_do_not_change_a_job(gpu_ctx, scenes_, w, h, exact):  # noqa: F811
    job = _job(scenes_[1], w, h, 6, 2)
    alone, st = _run(gpu_ctx, [job], exact=exact)
    mixed, _ = _run(gpu_ctx, [job, _job(scenes_[3], 300, 200, 6, 2)], exact=exact)
    assert st["samples"] == 2 * w * h
    assert np.array_equal(alone[0].view(np.int32), mixed[0].view(np.int32))
    if w > 30:
        assert alone[0][:, 3].sum() > 0
