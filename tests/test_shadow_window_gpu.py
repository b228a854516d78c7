"""The shadow visibility's 5 x 5 texel window (calc_visibility) against the oracle's sixteen separate taps, at map
sizes smaller than the window, odd, and large, so that windows straddle every border of the map and lie outside it:
the deterministic injection's RGBA8 averages and the octree's fragment colours are equal word for word."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)


@pytest.mark.parametrize("width,height", [(1, 1), (4, 3), (5, 5), (7, 64), (250, 33), (2048, 2048)])
def test_window_equals_sixteen_taps(cuda, oracle, width, height):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import room_scene
    scene = room_scene(seed=4, n_random=1500)
    ds, ws, R = passes.DeviceScene(scene), passes.Workspace(), 32
    shadow = np.random.default_rng(width).random((height, width), dtype=np.float32)
    tsh = torch.from_numpy(shadow).cuda()
    # the map covers +-16 units around the origin's ray: a far one leaves part of the room outside
    for origin in ((0.0, 15.0, 0.0), (9.0, 15.0, -14.0)):
        sd = passes.light_shadow_desc(origin, LIGHT_DIR)
        regions = clipmap.clip_regions((0.0, 4.0, 0.0), R)
        want = oracle.inject_radiance(scene, R, clipmap.regions_to_numpy(regions), shadow, bytes(sd))
        atlas = clipmap.new_atlas(R)
        passes.inject_radiance(ds, regions, R, tsh, passes.light_desc(LIGHT_DIR), sd, atlas, ws)
        assert np.array_equal(atlas.cpu().numpy().view(np.uint32), want)
        frags = passes.svo_fragments(ds, 6, tsh, passes.light_desc(LIGHT_DIR), sd, ws)
        fo, n = oracle.svo_fragments(scene, 6, ds.bb_min, ds.bb_max, shadow, bytes(sd))
        assert np.array_equal(frags.cpu().numpy().view(np.uint32), fo[:n])
