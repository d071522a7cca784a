"""Renders whose work items fill the default slot pool in one pass, several
passes of a smaller pool, and the first and later checks of the counters
(iterations launched one by one, then as graphs): the image, the path count
and the ray counts do not depend on any of it."""
import numpy as np
import pytest

from vviewer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,samples,depth,batch", [(1, 1, 1, 1, 1), (17, 3, 4, 2, 4), (640, 480, 16, 6, 4)])
def test_pool_size_and_check_interval_do_not_change_the_image(ctx, w, h, samples, depth, batch):
    e, info = scenes.cornell_box(11, w, h, samples, depth, batch)
    sd = e.scene.scene_data(w, h)
    g = ctx.upload(e.scene.build())
    ref, counts = None, None
    try:
        for slots, iterations in ((0, 0), (0, 1), (0, 64), (1 << 20, 8), (4096, 2)):
            ctx.set_tuning(slots=slots, iterations_per_graph=iterations)
            r = g.render(sd, info)
            s = ctx.stats()
            now = (s.paths, s.segments, s.shadow_rays, s.emitter_rays)
            if ref is None:
                ref, counts = r, now
            for k in ("radiance", "albedo", "normal"):
                assert np.array_equal(getattr(r, k), getattr(ref, k)), (slots, iterations, k)
            assert now == counts, (slots, iterations)
    finally:
        ctx.set_tuning()
        g.release()
