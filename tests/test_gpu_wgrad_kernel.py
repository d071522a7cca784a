"""The weight and bias gradient kernel on its own, both instantiations (64
input channels a block for 64, 112 and 128, else 32), against 64-bit sums of
the same BF16 inputs."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from vviewer_gb300 import build as vbuild

pytestmark = pytest.mark.gpu
HARNESS = Path(__file__).resolve().parent / "device_wgrad" / "device_wgrad.cu"
OUT = Path(__file__).resolve().parent / "_build" / "libdevice_wgrad.so"


@pytest.fixture(scope="module")
def wgrad():
    OUT.parent.mkdir(exist_ok=True)
    cmd = [vbuild._nvcc(), *vbuild.ARCH, *vbuild.NVCC_FLAGS, "-shared", str(HARNESS),
           str(vbuild.CSRC / "denoise_kernels.cu"), "-o", str(OUT)]
    subprocess.run(cmd, check=True, capture_output=True)
    lib = C.CDLL(str(OUT))
    lib.device_wgrad.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p,
                                 C.c_int]
    import torch

    def run(dout, x):
        n, h, w, cout = dout.shape
        cin = x.shape[3]
        weights = 9 * cin * cout
        g = torch.zeros((4, weights + cout), device="cuda")
        torch.cuda.synchronize()
        assert lib.device_wgrad(dout.data_ptr(), cout, x.data_ptr(), cin, n, h, w, g.data_ptr(), g.shape[1]) == 0
        return g[0, :weights].reshape(cout, 3, 3, cin), g[0, weights:]

    return run


# Whole numbers from -3 to 3: every sum stays below 2^24, so the gradients are
# exact in any order of the additions.
@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 16), (80, 32), (96, 96), (160, 64), (224, 96), (64, 64),
                                      (112, 48), (128, 128)])
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (3, 2, 15), (1, 5, 63), (2, 3, 64), (1, 4, 65), (1, 17, 272)])
def test_gradients_of_whole_numbers_are_exact(wgrad, n, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n * 1000 + w + cin)
    dout = torch.randint(-3, 4, (n, h, w, cout), generator=g, device="cuda").double()
    x = torch.randint(-3, 4, (n, h, w, cin), generator=g, device="cuda").double()
    dw, db = wgrad(dout.bfloat16(), x.bfloat16())
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    want = torch.stack([torch.stack([torch.einsum("nhwo,nhwi->oi", dout, xp[:, i:i + h, j:j + w]) for j in range(3)], 1)
                        for i in range(3)], 1)
    assert torch.equal(dw.double(), want)
    assert torch.equal(db.double(), dout.sum((0, 1, 2)))


# The bias gradient is summed in FP32, each addition rounded to nearest: its
# errors have no preferred sign. A sum passes through at most 16 additions (a
# row's 64 pixels by halves, the 8 rows' sums, the copies), every one off by at
# most 2^-24 of the result, evenly distributed (an rms of 2^-24 / sqrt(3)): the
# mean over all channels and draws lies within 6 standard deviations of zero.
# Sums that are cut off instead of rounded are below the exact ones on average.
@pytest.mark.parametrize("cin", [32, 64])
def test_bias_gradient_rounds_to_nearest(wgrad, cin):
    import torch
    g = torch.Generator(device="cuda").manual_seed(cin)
    errors = []
    for _ in range(32):
        dout = torch.rand((1, 8, 64, 128), generator=g, device="cuda") + 1.0
        dout *= torch.exp2(-torch.randint(0, 17, dout.shape, generator=g, device="cuda").float())
        dout = dout.bfloat16()
        _, db = wgrad(dout, torch.zeros((1, 8, 64, cin), device="cuda", dtype=torch.bfloat16))
        exact = dout.double().sum((0, 1, 2))
        errors.append((db.double() - exact) / exact * 2.0 ** 24)
    e = torch.cat(errors)
    assert abs(float(e.mean())) <= 6.0 * (16 / 3) ** 0.5 / e.numel() ** 0.5, (float(e.mean()), float(e.std()))
