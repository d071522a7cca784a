"""Denoisers of several threads, each with a context of its own, whose first
calls come at once and need different amounts of shared memory: the same
images as one after the other. In a process of its own, where no call has set
up a kernel before."""
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CHILD = textwrap.dedent("""
    import sys, threading
    sys.path.insert(0, sys.argv[1])
    import torch
    from vviewer_gb300 import Context
    from vviewer_gb300.denoiser import Denoiser
    SIZES = [(16, 16), (64, 48), (256, 256), (480, 272), (1024, 512), (128, 1024), (32, 512), (1920, 1088)]
    work = []
    for k, (w, h) in enumerate(SIZES):
        g = torch.Generator(device="cuda").manual_seed(k)
        work.append((Denoiser(Context(0), seed=3), [torch.rand((h, w, 4), generator=g, device="cuda") for _ in range(3)],
                     torch.zeros((h, w, 4), device="cuda")))
    torch.cuda.synchronize()
    start, failed = threading.Barrier(len(work)), []

    def run(dn, images, out):
        start.wait()
        try:
            dn.apply(*images, out)
            if images[0].shape[0] <= 272:
                dn.gradients(*[x[None] for x in images], images[0][None])
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=run, args=a) for a in work]
    for t in threads: t.start()
    for t in threads: t.join()
    assert not failed, failed
    for dn, images, out in work:
        again = torch.zeros_like(out)
        dn.apply(*images, again)
        torch.cuda.synchronize()
        assert torch.equal(out, again), out.shape
""")


def test_first_calls_of_several_threads(tmp_path):
    script = tmp_path / "child.py"
    script.write_text(CHILD)
    run = subprocess.run([sys.executable, str(script), str(ROOT)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-3000:]
