"""Where vvpt_trace_closest stores a device caller's hits: in an array of its
own, over the rays themselves (from their start, in their middle, over their
end), and at an address that is not aligned. Below and above the batch size
from which the kernel refills its lanes (five blocks of 256 rays per SM)."""
import numpy as np
import pytest

from raygen import HIT_SCENES, make_rays
from vviewer_gb300.renderer import HIT_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1001, 250_001])
def test_hits_over_the_rays(ctx, n):
    import torch
    build, (lo, hi) = HIT_SCENES["cornell"]
    flat = build().scene.build()
    rays = np.ascontiguousarray(make_rays(flat, n, 5, lo, hi)[:n], dtype=np.float32)
    gpu = ctx.upload(flat)
    want = gpu.trace_closest(rays).view(np.uint8)
    raw = torch.from_numpy(rays).view(torch.uint8).reshape(-1).cuda()
    at_rays, size = 64, HIT_DTYPE.itemsize * n
    for at in (at_rays + 32 * n + 4, at_rays, at_rays + 32 * (n // 2), at_rays + 32 * n - 4, at_rays + 32 * n + 2, 0):
        buf = torch.zeros(at_rays + 64 * n + 64, dtype=torch.uint8, device="cuda")
        buf[at_rays:at_rays + 32 * n] = raw
        torch.cuda.synchronize()
        p = buf.data_ptr()
        ctx.check(ctx.lib.vvpt_trace_closest(ctx.handle, gpu.handle, p + at_rays, n, p + at, 1))
        got = buf[at:at + size].cpu().numpy()
        assert np.array_equal(got, want), at
    gpu.release()
