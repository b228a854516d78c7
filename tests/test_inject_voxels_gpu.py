"""The injection's grouping by voxel (runs of samples, sorted by voxel, folded by eight lanes or, past 64 runs, by a
block) against the oracle's serial fold, bit for bit: small grids put thousands of samples on one voxel, larger ones
a few; atlases empty and prefilled (alpha chains that wrap), emissive triangles that write all six faces, every level
and a subset."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)


@pytest.mark.parametrize("R,mask", [(8, 0x3F), (16, 0x3F), (32, 0x15), (64, 0x3F)])
@pytest.mark.parametrize("prefilled", [False, True])
def test_fold_equals_the_oracle(cuda, oracle, R, mask, prefilled):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import room_scene
    scene = room_scene(seed=6, n_random=6000)
    scene.materials["emissive_factor"][::5] = (0.25, 1.2, 0.0)
    scene.textures[::3] &= 0xff00ffff  # zero channels
    ds, ws = passes.DeviceScene(scene), passes.Workspace()
    regions = clipmap.clip_regions((0.5, 3.0, -0.4), R)
    origin = (-4.0, 16.0, -3.0)
    sd = passes.light_shadow_desc(origin, LIGHT_DIR)
    shadow = np.random.default_rng(R).random((128, 96), dtype=np.float32)
    shadow[shadow < 0.4] = 0.0
    atlas = np.zeros(((R + 2), 6 * (R + 2), 6 * (R + 2)), np.uint32)
    if prefilled:
        atlas = np.random.default_rng(R + 1).integers(0, 1 << 32, atlas.shape, dtype=np.uint64).astype(np.uint32)
        atlas[::2] &= 0x00ffffff  # alpha 0 under a colour
    t = torch.from_numpy(atlas.view(np.int32).copy()).cuda()
    passes.inject_radiance(ds, regions, R, torch.from_numpy(shadow).cuda(), passes.light_desc(LIGHT_DIR), sd, t, ws,
                           level_mask=mask)
    want = oracle.inject_radiance(scene, R, clipmap.regions_to_numpy(regions), shadow, bytes(sd), level_mask=mask,
                                  atlas=atlas)
    got = t.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, want), np.count_nonzero(got != want)


def test_more_than_2_27_samples_take_wide_runs(cuda):
    """45 stacked quads larger than the grid cover about 144M samples over six levels of 256^3 (64-bit runs); each
    level on its own stays below 2^27 (32-bit runs).  Levels do not share voxels, so the atlases are equal."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import _pack
    R, big = 256, 2000.0
    rng = np.random.default_rng(9)
    quads = []
    for i in range(45):
        y = np.float32(4.0 + 0.01 * i)
        a, b, c, d = [-big, y, -big], [big, y, -big], [big, y, big], [-big, y, big]
        quads += [[a, c, b], [a, d, c]]
    ds, ws = passes.DeviceScene(_pack(np.array(quads, np.float32), rng)), passes.Workspace()
    regions, light = clipmap.clip_regions((0.0, 4.0, 0.0), R), passes.light_desc(LIGHT_DIR)
    sd = capi.DirectionalLightShadowDesc()
    whole, parts = clipmap.new_atlas(R), clipmap.new_atlas(R)
    passes.inject_radiance(ds, regions, R, None, light, sd, whole, ws)
    assert ws.nbytes > 32 * (1 << 27)  # the descriptors alone
    for l in range(6):
        passes.inject_radiance(ds, regions, R, None, light, sd, parts, ws, level_mask=1 << l)
    assert torch.equal(whole, parts) and int((whole != 0).sum().item()) > 100000
    ws.close()
