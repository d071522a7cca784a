"""Device memory that plain renders keep: by default one path slot of 304
bytes per work item; within a budget fewer, with the same image; given back
when a budget or a smaller number of slots is set."""
import numpy as np
import pytest

from vviewer_gb300 import Context, scenes

pytestmark = pytest.mark.gpu


def test_pool_is_bounded_and_given_back():
    import torch
    e, info = scenes.cornell_box(2, 1600, 1200, 4, 3, 1)
    items = 1600 * 1200 * 4
    sd = e.scene.scene_data(1600, 1200)
    ctx = Context(0)
    g = ctx.upload(e.scene.build())
    out = {k: torch.zeros((1200, 1600, 4), device="cuda") for k in ("radiance", "albedo", "normal")}
    torch.cuda.synchronize()

    def held():
        return start - torch.cuda.mem_get_info()[0]

    def render():
        g.render(sd, info, outputs={k: v.data_ptr() for k, v in out.items()})
        return {k: v.cpu().numpy() for k, v in out.items()}

    slack = 16 << 20  # allocation granularity
    ctx.set_tuning(slots=4096)
    ref = render()
    ctx.set_tuning()
    start = torch.cuda.mem_get_info()[0]
    images = [render()]
    full = held()
    assert abs(full - 304 * (items - 4096)) < slack
    ctx.set_tuning(slots=1 << 20)
    assert held() <= slack  # given back
    images.append(render())
    assert held() <= 304 * (1 << 20) + slack
    ctx.set_tuning()
    images.append(render())
    assert abs(held() - full) < slack
    ctx.set_budget(1 << 30)
    assert held() <= slack
    images.append(render())
    assert 304 * (1 << 20) - slack <= held() <= (1 << 30) + slack
    ctx.set_budget(0)
    images.append(render())
    assert abs(held() - full) < slack
    for im in images:
        for k in ref:
            assert np.array_equal(im[k], ref[k]), k
    g.release()
    ctx.close()
    assert held() <= slack
