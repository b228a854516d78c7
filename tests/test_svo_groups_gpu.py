"""The octree's specular cones by eight lanes, four, two and one over several pools and decays: pools that stop the
cones early and late, decays that add little and much, all specular and some."""
import numpy as np
import pytest

from .test_svo_trace_rules import dense_pool

pytestmark = pytest.mark.gpu

BOX = ((-4.0, -4.0, -4.0), (4.0, 4.0, 4.0))
EYE = (0.0, 1.0, -4.0)


@pytest.mark.parametrize("depth,fill,decay,fraction", [(6, 0.9, 0.0, 1.0), (5, 0.4, 3.0, 1.0), (3, 0.7, 0.05, 0.3),
                                                       (6, 0.2, 0.0, 0.6)])
def test_groups_equal_one_lane_and_the_oracle(cuda, oracle, depth, fill, decay, fraction):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import random_samples
    pool_np = dense_pool(depth, 11, fill)
    pool = torch.from_numpy(pool_np.view(np.int32).copy()).cuda()
    desc = clipmap.trace_desc(volume_center=[0.0, 0.0, 0.0], rendering_mode=8, voxel_size=0.125, volume_dimension=64.0,
                              trace_start_offset=1.0, indirect_diffuse_intensity=8.0, ambient_occlusion_factor=0.5,
                              min_trace_step_factor=1.0, indirect_specular_intensity=3.0, occlusion_decay=decay,
                              enable_32_cones=0)
    rec = random_samples(400, (0, 0, 0), 3.0, seed=depth, specular_fraction=fraction)
    want_d, want_s, want_steps = oracle.svo_trace(32, bytes(desc), EYE, pool_np, rec, *BOX)
    few, first = clipmap.samples_to_device(rec), None
    # 400 samples to 432,000, of which up to 311,296 lanes' worth of cones (any grid's) take more than one lane
    for times in (1, 40, 130, 270, 1080):
        steps = torch.zeros(1, dtype=torch.int64, device="cuda")
        d, s = passes.svo_cone_trace(desc, EYE, pool, pool.shape[0], few.repeat(times, 1), *BOX, steps=steps)
        if first is None:
            first = d, s, int(steps.item())
        assert int(steps.item()) == first[2] * times, times
        for got, w in ((d, first[0]), (s, first[1])):
            assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(w.repeat(times, 1))), times
    for got, want in ((first[0], want_d), (first[1], want_s)):
        got = np.nan_to_num(got.cpu().numpy())
        want = np.nan_to_num(want)
        err = np.abs(got - want).max(1) / np.maximum(np.abs(want).max(1), 1e-3)
        assert np.mean(err < 1e-4) > 0.99, np.sort(err)[-8:]  # as the dense pools' bar
    assert abs(first[2] - want_steps) <= max(8, 0.002 * want_steps)
