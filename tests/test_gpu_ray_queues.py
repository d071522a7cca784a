"""The kinds of ray one trace launch takes (extension, shadow, emitter rays of
ended paths, and what is left to the candidate walk) against the oracle, and
the same image for every split of the work: one warp of slots, a ragged
number, more slots than work items."""
import numpy as np
import pytest

from oracle import oracle
from test_gpu_parity import compare_renders
from vviewer_gb300 import scenes

pytestmark = pytest.mark.gpu


# zfar beyond the extension rays' range (10000): a continuing path's emitter
# ray is a ray of its own. The bounds are the parity suite's for a render
# against the oracle.
@pytest.mark.parametrize("zfar", [50.0, 20000.0])
@pytest.mark.parametrize("depth", [1, 2, 9])
def test_rays_of_a_medium_scene_match_oracle(ctx, depth, zfar):
    engine, info = scenes.cornell_medium(3, 48, 32, 16, depth, 4, freq=6)
    engine.scene.camera.zfar = zfar
    flat, sd = engine.scene.build(), engine.scene.scene_data(info.width, info.height)
    gpu = ctx.upload(flat)
    images = []
    for slots in (0, 32, 1000, 1 << 16):
        ctx.set_tuning(slots=slots)
        images.append(gpu.render(sd, info, want_m2=True))
    ctx.set_tuning()
    gpu.release()
    for other in images[1:]:
        assert np.array_equal(images[0].radiance, other.radiance)
        assert images[0].stats.shadow_rays == other.stats.shadow_rays
        assert images[0].stats.emitter_rays == other.stats.emitter_rays
    ref = oracle.render(flat, sd, info)
    rel, close, z4 = compare_renders(images[0].radiance, ref["radiance"], images[0].radiance_m2, 4)
    assert rel < 1e-4 and close >= 0.95 and z4 < 0.005, (rel, close, z4)
