"""Meshes that the GPU builder takes in several groups (scenes of more than
VVPT_GROUP_TRIANGLES triangles): the library is built a second time, in-tree,
with groups of at most 700 triangles, and driven from a child process. Closest
hits equal to the oracle's; the scene's arrays hold every group's meshes, a
mesh larger than a group, and what the host adds (a small mesh, baked
instances)."""
import subprocess
import sys
import textwrap
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle
from raygen import make_rays
from test_gpu_bvh_sizes import _triangles
from vviewer_gb300.scene import Engine, MaterialLambert, Transform
from vviewer_gb300.scenes import mesh_from_triangles

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
SIZES = (512, 40, 600, 2000, 12, 513, 100, 700, 3, 30)

CHILD = textwrap.dedent("""
    import sys
    import numpy as np
    sys.path[:0] = [sys.argv[3], sys.argv[3] + "/tests"]
    from vviewer_gb300 import _native as N
    N.load(sys.argv[1])
    from vviewer_gb300 import Context
    import test_gpu_mesh_groups as T
    ctx = Context(0)
    flat, rays = T.scene()
    gpu = ctx.upload(flat)
    np.save(sys.argv[2], gpu.trace_closest(rays))
    gpu.release()
    ctx.close()
""")


def scene():
    rng = np.random.default_rng(8)
    engine = Engine()
    mat = engine.create_material(MaterialLambert, "m")
    for k, n in enumerate(SIZES):
        mesh = engine.add_mesh(mesh_from_triangles(f"m{k}", _triangles("random", n, rng)))
        for j in range(1 + k % 2):
            so = engine.scene.add_scene_object(f"o{k}_{j}", Transform((0.3 * k, 0.9 * j, 0.0)))
            so.mesh, so.material = mesh, mat
    flat = engine.scene.build()
    return flat, make_rays(flat, 20_000, 3, -0.5, 4.0)


def test_hits_of_grouped_meshes_match_oracle(ctx, tmp_path):
    from vviewer_gb300 import build as B
    lib = B.build(force=True, defines=["VVPT_GROUP_TRIANGLES=700"], out=B.OUT_DIR / "variants" / "libvvpt_groups.so",
                  build_dir=B.BUILD_DIR / "groups")
    res, script = tmp_path / "hits.npy", tmp_path / "child.py"
    script.write_text(CHILD)
    run = subprocess.run([sys.executable, str(script), str(lib), str(res), str(ROOT)], capture_output=True, text=True,
                         timeout=600)
    assert run.returncode == 0, run.stderr[-4000:]
    flat, rays = scene()
    want = oracle.trace_closest(flat, rays)
    got = np.load(res)
    gpu = ctx.upload(flat)
    one = gpu.trace_closest(rays)
    gpu.release()
    assert (want["instance"] != 0xFFFFFFFF).mean() > 0.3
    for f in ("instance", "primitive", "t", "u", "v"):
        assert np.array_equal(got[f], want[f]), f
        assert np.array_equal(one[f], want[f]), f
