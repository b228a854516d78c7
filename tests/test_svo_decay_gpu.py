"""Octree cones under occlusion decays whose divisor 1 + (step + size) * decay vanishes or is NaN: a step through
empty nodes then ends the march (0 / 0), as in the shader's loop, whether one lane marches a cone or several do."""
import numpy as np
import pytest

from .test_svo_trace_rules import dense_pool

pytestmark = pytest.mark.gpu

BOX = ((-4.0, -4.0, -4.0), (4.0, 4.0, 4.0))
EYE = (0.0, 1.0, -4.0)


def make_desc(clipmap, mode, decay, voxel):
    return clipmap.trace_desc(volume_center=[0.0, 0.0, 0.0], rendering_mode=mode, voxel_size=voxel,
                              volume_dimension=8.0 / voxel, trace_start_offset=1.0, indirect_diffuse_intensity=8.0,
                              ambient_occlusion_factor=0.5, min_trace_step_factor=1.0,
                              indirect_specular_intensity=3.0, occlusion_decay=decay, enable_32_cones=0)


# every sample lies within half of level 0's radius, so its cones' first step is of one level-0 voxel: with a decay of
# -1 / voxel the divisor is exactly 0 there
@pytest.mark.parametrize("voxel,decay", [(0.25, -4.0), (0.5, -2.0), (0.25, float("nan"))])
@pytest.mark.parametrize("mode", [5, 6])  # the diffuse cones' colour, the specular cone's
def test_vanishing_divisor_ends_the_march(cuda, oracle, voxel, decay, mode):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import random_samples
    pool_np = dense_pool(4, 7)
    pool = torch.from_numpy(pool_np.view(np.int32).copy()).cuda()
    desc = make_desc(clipmap, mode, decay, voxel)
    rec = random_samples(600, (0, 0, 0), 1.0, seed=6, specular_fraction=1.0)
    rec = rec[np.linalg.norm(rec["position"], axis=1) < 1.5]
    want_d, want_s, want_steps = oracle.svo_trace(32, bytes(desc), EYE, pool_np, rec, *BOX)
    few = clipmap.samples_to_device(rec)
    for times in (1, 1100):  # eight lanes to a specular cone, then one
        steps = torch.zeros(1, dtype=torch.int64, device="cuda")
        d, s = passes.svo_cone_trace(desc, EYE, pool, pool.shape[0], few.repeat(times, 1), *BOX, steps=steps)
        assert int(steps.item()) == want_steps * times, (times, int(steps.item()), want_steps)
        n = rec.shape[0]
        for got, want in ((d, want_d), (s, want_s)):
            got = got.cpu().numpy().reshape(times, n, 4)
            assert np.array_equal(got, np.broadcast_to(got[:1], got.shape))
            err = np.abs(got[0, :, :3] - want[:, :3]).max(1) / np.maximum(np.abs(want[:, :3]).max(1), 1e-3)
            assert np.mean(err < 1e-4) > 0.99, np.sort(err)[-8:]
