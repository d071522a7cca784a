"""The denoiser's convolutions over image sizes that change how a layer is
split: all output channels in a CTA or a share of them (small images), one or
two sets of drain warps, fused upsample + concat inputs at one CTA per SM,
segments shorter and longer than the ring, partial 128-pixel columns, 2x2 averages written by
the drains, layers whose weights are shared out over two CTAs (from one row of 128 pixels per SM). The split
changes which CTA adds up an output element, not the order of its sum: the
image is bit-identical between the strip kernel's plans and with the unfused
inputs. Against the mma.sync kernels, whose sums run in another order before
the same BF16 roundings, the bound is the one the per-kernel test has (rtol
2e-2, atol 1e-3)."""
import numpy as np
import pytest

from test_gpu_denoiser import _cuda
from vviewer_gb300.denoiser import Denoiser

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(16, 16), (16, 272), (144, 16), (128, 128), (256, 256), (272, 400), (544, 976), (1072, 1104)])
def test_split_does_not_change_the_image(ctx, h, w):
    import torch
    rng = np.random.default_rng(h * 10000 + w)
    ins = [_cuda(rng.gamma(1.0, 0.5, (h, w, 4))), _cuda(rng.uniform(0, 1, (h, w, 4))),
           _cuda(rng.uniform(0, 1, (h, w, 4)))]
    dn = Denoiser(ctx, seed=9)
    outs = {}
    for kind in ("tcgen05", "tcgen05_unfused", "tcgen05_persistent", "mma_sync"):
        dn.set_kernels(kind)
        o = torch.zeros((h, w, 4), device="cuda")
        dn.apply(*ins, o)
        torch.cuda.synchronize()
        outs[kind] = o.cpu().numpy()
    dn.close()
    assert np.array_equal(outs["tcgen05"], outs["tcgen05_unfused"])
    assert np.array_equal(outs["tcgen05"], outs["tcgen05_persistent"])
    np.testing.assert_allclose(outs["tcgen05"], outs["mma_sync"], rtol=2e-2, atol=1e-3)
