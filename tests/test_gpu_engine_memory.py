"""The job engine's fixed device memory: 300 bytes a path slot (a path's
members 252, its places in the queues 44, in the idle list 4), which a budget
set by callers leaves beside the jobs. A job is admitted at that budget."""
import numpy as np
import pytest

from vviewer_gb300 import Context, scenes

pytestmark = pytest.mark.gpu


def test_fixed_bytes_per_slot_and_admission():
    fixed = {}
    e, info = scenes.cornell_box(4, 64, 48, 8, 4, 4)
    for slots in (1 << 18, 1 << 20):
        ctx = Context(0)
        ctx.set_tuning(slots=slots)
        fixed[slots] = ctx.engine_stats().fixed_bytes
        if slots == 1 << 20:
            per_job = 3 * 16 * 64 * 48 * 2 + 3 * 16 * 64 * 48  # batch sums, staged images
            ctx.set_budget(fixed[1 << 18] + 300 * ((1 << 20) - (1 << 18)) + per_job)
            g = ctx.upload(e.scene.build())
            sd = e.scene.scene_data(64, 48)
            job = g.submit(sd, info)
            got = job.result().radiance
            assert np.array_equal(got, g.render(sd, info).radiance)
            job.release()
            g.release()
        ctx.close()
    assert fixed[1 << 20] - fixed[1 << 18] <= 300 * ((1 << 20) - (1 << 18))
