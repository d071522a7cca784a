"""A denoiser's calls after one that found no device memory for its buffers,
on a device of the test's own: the same call fails again instead of running
on buffers that are not there, and succeeds once there is room; an image call
needs no more than its own buffers after a failed training call."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "vviewer_gb300" / "csrc"
HARNESS = Path(__file__).resolve().parent / "host_denoiser" / "host_denoiser.cpp"
OUT = Path(__file__).resolve().parent / "_build" / "libhost_denoiser.so"
APPLY, GRADS = 0, 1
OK, OOM = 0, 2


@pytest.fixture(scope="module")
def calls():
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                 if p and (Path(p) / "include" / "vector_types.h").exists()), None)
    if not cuda:
        pytest.skip("CUDA headers (vector_types.h) not found")
    OUT.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-pthread", "-Wl,-Bsymbolic", "-I",
                    f"{cuda}/include", "-I", str(ROOT / "include"), "-I", str(CSRC), str(HARNESS), "-x", "c++",
                    str(CSRC / "denoise.cu"), "-o", str(OUT)], check=True, capture_output=True)
    lib = C.CDLL(str(OUT))

    def run(*todo):
        n = len(todo)
        cols = [(C.c_int * n)(*[t[k] for t in todo]) for k in range(4)]
        status, bad = (C.c_int * n)(*[-1] * n), (C.c_int * n)()
        lib.host_denoiser_calls(n, *cols, status, bad)
        assert list(bad) == [0] * n, list(bad)
        return list(status)

    return run


@pytest.mark.parametrize("kind", [APPLY, GRADS])
def test_the_same_call_fails_again_until_there_is_room(calls, kind):
    assert calls((kind, 64, 64, 1), (kind, 64, 64, 1), (kind, 64, 64, 64), (kind, 64, 64, 0)) == [OOM, OOM, OK, OK]


def test_a_failed_larger_call_leaves_the_denoiser_usable(calls):
    # 64 x 64: 3.3 MB of activations and 0.3 MB of output for an image; 128 x 128
    # with gradients needs 42 MB
    assert calls((APPLY, 64, 64, 8), (GRADS, 128, 128, 2), (APPLY, 64, 64, 8), (GRADS, 128, 128, 2), (APPLY, 128, 128, 24),
                 (GRADS, 128, 128, 64), (APPLY, 64, 64, 0)) == [OK, OOM, OK, OOM, OK, OK, OK]
