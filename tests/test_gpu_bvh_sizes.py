"""The GPU tree builder at the sizes where its forms meet (a leaf, one warp's
range, the first levels, the size that leaves the host builder) and on meshes
that no plane separates: closest hits equal to the oracle's, several meshes in
one build."""
import numpy as np
import pytest

from oracle import oracle
from raygen import make_rays
from test_gpu_parity import N_BVH_AUTO, N_BVH_GPU, assert_hits_equal
from vviewer_gb300.scene import Engine, MaterialLambert, Transform
from vviewer_gb300.scenes import mesh_from_triangles

pytestmark = pytest.mark.gpu


def _triangles(kind, n, rng):
    p = rng.uniform(0, 1, (n, 1, 3)) + rng.normal(0, 0.05, (n, 3, 3))
    if kind == "equal":  # one triangle n times: every centroid the same
        p[:] = p[0]
    elif kind == "flat":  # all in one plane, centroids on a line
        p[..., 2] = 0.25
        p[..., 1] -= p[..., 1].mean(1, keepdims=True)
    return p.reshape(-1, 3).astype(np.float32)


@pytest.mark.parametrize("kind", ["random", "equal", "flat", "nan"])
@pytest.mark.parametrize("sizes", [(5, 65), (31, 32, 33), (66, 256, 257), (511, 512, 513, 2000)])
def test_hits_match_oracle(ctx, kind, sizes):
    rng = np.random.default_rng(sum(sizes))
    engine = Engine()
    mat = engine.create_material(MaterialLambert, "m")
    for k, n in enumerate(sizes):
        so = engine.scene.add_scene_object(f"o{k}", Transform((0.3 * k, 0.0, 0.0)))
        so.mesh = engine.add_mesh(mesh_from_triangles(f"m{k}", _triangles(kind, n, rng)))
        if kind == "nan":  # some triangles without a box
            so.mesh.vertices["position"].reshape(n, 3, 3)[:: max(2, n // 5)] = np.nan
        so.material = mat
    flat = engine.scene.build()
    rays = make_rays(flat, 20_000, 3, -0.5, 2.0)
    rays = rays[np.isfinite(rays).all(1)]
    want = oracle.trace_closest(flat, rays)
    try:
        for builder in (N_BVH_GPU, N_BVH_AUTO):
            ctx.check(ctx.lib.vvpt_set_bvh_builder(ctx.handle, builder))
            gpu = ctx.upload(flat)
            assert_hits_equal(gpu.trace_closest(rays), want)
            gpu.release()
    finally:
        ctx.check(ctx.lib.vvpt_set_bvh_builder(ctx.handle, N_BVH_AUTO))
