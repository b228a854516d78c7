"""The shadow visibility of positions that project far outside the map -- past 2^22 texels, where consecutive texel
indices stop being distinct floats, and past 2^31, where they leave the integers -- is the sixteen taps': the oracle's,
or none lit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)


@pytest.mark.parametrize("width,height", [(64, 64), (333, 5)])
def test_far_positions_equal_sixteen_taps(cuda, oracle, width, height):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import room_scene
    scene, R = room_scene(seed=4, n_random=800), 32
    scene.materials["emissive_factor"] = 0.0  # only visible surfaces add light
    ds, ws = passes.DeviceScene(scene), passes.Workspace()
    shadow = np.random.default_rng(width).random((height, width), dtype=np.float32)
    tsh = torch.from_numpy(shadow).cuda()
    regions = clipmap.clip_regions((0.0, 4.0, 0.0), R)
    reg = clipmap.regions_to_numpy(regions)
    lit = []
    # the map is 32 units wide: a scale of 2^k puts a unit at width / 32 * 2^k texels
    for kx, ky in ((0, 0), (6, 0), (16, 0), (0, 21), (20, 1), (27, 0), (0, 28), (29, 0), (30, 30), (32, 0), (0, 40), (90, 0)):
        sd = passes.light_shadow_desc((0.0, 15.0, 0.0), LIGHT_DIR)
        sd.proj[0] *= 2.0 ** kx
        sd.proj[5] *= 2.0 ** ky
        atlas = clipmap.new_atlas(R)
        passes.inject_radiance(ds, regions, R, tsh, passes.light_desc(LIGHT_DIR), sd, atlas, ws)
        got = atlas.cpu().numpy().view(np.uint32)
        if max(kx, ky) < 27:  # the oracle's own indices are integers here
            want = oracle.inject_radiance(scene, R, reg, shadow, bytes(sd))
            assert np.array_equal(got, want), (kx, ky)
            lit.append(int(np.count_nonzero(want)))
        else:  # no position lies within the map, whose border is unlit
            assert not got.any(), (kx, ky)
    assert lit[0] > 1000 and 0 < lit[1] < lit[0] and min(lit) < lit[0] // 50, lit
