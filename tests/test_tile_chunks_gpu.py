"""The coverage kernels' chunks take tiles from all over the list by its length (fewer than 2^18 tiles, 2^20, more):
opacity, the deterministic injection and the octree's fragment list stay equal to the oracle's (or, for the longest
list, to the same triangles rasterised in two halves)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)


@pytest.mark.parametrize("R,n_random", [(16, 0), (64, 3), (64, 9000), (256, 2500)])
def test_opacity_and_injection_equal_the_oracle(cuda, oracle, R, n_random):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import room_scene
    scene = room_scene(seed=8, n_random=n_random)
    ds, ws = passes.DeviceScene(scene), passes.Workspace()
    regions = clipmap.clip_regions((0.3, 2.5, -0.4), R)
    rn = clipmap.regions_to_numpy(regions)
    mask = 0x3F if R < 256 else 0x24
    want = oracle.voxelize_opacity(scene, R, rn, level_mask=mask)
    atlas = clipmap.new_atlas(R)
    passes.voxelize_opacity(ds, regions, R, atlas, ws, level_mask=mask)
    assert np.array_equal(atlas.cpu().numpy().view(np.uint32), want)
    atlas.zero_()
    passes.inject_radiance(ds, regions, R, None, passes.light_desc(LIGHT_DIR), capi.DirectionalLightShadowDesc(), atlas,
                           ws, level_mask=mask)
    want = oracle.inject_radiance(scene, R, rn, None, bytes(capi.DirectionalLightShadowDesc()), level_mask=mask)
    assert np.array_equal(atlas.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("triangles", [1, 20, 90000, 700000, 1300000])
def test_fragment_list_is_its_halves(cuda, triangles):
    """The list of a scene is the list of its first triangles followed by that of the rest."""
    torch = cuda
    import copy
    from vk_voxel_cone_tracing_gb300 import capi, passes
    from vk_voxel_cone_tracing_gb300.scene import terrain_scene
    scene = terrain_scene(seed=5, target=max(triangles, 40), boxes=triangles // 300)
    T, ws, sd = scene.indices.shape[0], passes.Workspace(), capi.DirectionalLightShadowDesc()
    whole = passes.DeviceScene(scene)
    lists = []
    for lo, hi in ((0, T), (0, T // 3), (T // 3, T)):
        part = copy.copy(scene)
        part.indices, part.tri_material = scene.indices[lo:hi], scene.tri_material[lo:hi]
        if hi > lo:
            lists.append(passes.svo_fragments(passes.DeviceScene(part), 8, None, passes.light_desc(LIGHT_DIR), sd, ws,
                                              bb_min=whole.bb_min, bb_max=whole.bb_max))
    assert torch.equal(lists[0], torch.cat(lists[1:]))


def test_edges_around_the_32_bit_limits(cuda, oracle):
    """Triangles with edges just below and above 2^17 (512 pixels of 1/256) and edge values past 2^31, fanned with
    shared edges, at one sample (shadow depth) and eight (opacity at R = 256)."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import _pack
    rng = np.random.default_rng(4)
    tris = []
    for size in (0.5, 3.9, 7.98, 8.0, 8.02, 15.9, 29.0, 300.0):
        c = rng.uniform(-3, 3, 3) + np.array([0.0, 4.0, 0.0])
        e = rng.normal(size=(2, 3))
        e = e / np.linalg.norm(e, axis=1, keepdims=True) * size
        a, b = c + e[0], c + e[1]
        tris += [[c, a, a + e[1]], [c, a + e[1], b], [c, b, c - e[0]]]
    scene = _pack(np.array(tris, np.float32), rng)
    ds, ws = passes.DeviceScene(scene), passes.Workspace()
    origin = (-4.0, 16.0, -3.0)
    depth = torch.empty((2048, 2048), dtype=torch.float32, device="cuda")
    passes.shadow_depth(ds, passes.light_shadow_desc(origin, LIGHT_DIR), depth, ws)
    want = oracle.shadow_depth(scene, oracle.light_shadow_desc(origin, LIGHT_DIR), 2048, 2048)
    assert np.array_equal(depth.cpu().numpy().view(np.uint32), want.view(np.uint32))
    R = 256
    regions = clipmap.clip_regions((0.0, 4.0, 0.0), R)
    atlas = clipmap.new_atlas(R)
    passes.voxelize_opacity(ds, regions, R, atlas, ws, level_mask=0x5)
    want = oracle.voxelize_opacity(scene, R, clipmap.regions_to_numpy(regions), level_mask=0x5)
    assert np.array_equal(atlas.cpu().numpy().view(np.uint32), want)


def test_triangles_about_the_depth_limits(cuda, oracle):
    """Triangles facing each axis at depths on both sides of each clip level's near and far limits, from an ulp to
    a voxel away, flat and tilted across: the ones culled as a whole leave the atlases the oracle's."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import _pack
    rng = np.random.default_rng(8)
    R = 32
    regions = clipmap.clip_regions((0.3, 1.2, -0.6), R)
    reg = clipmap.regions_to_numpy(regions)
    tris = []
    for level in (0, 2):
        vs = float(reg[level, 6:7].view(np.float32)[0])
        lo = reg[level, 0:3].astype(np.float64) * vs
        size = R * vs
        for axis in range(3):
            for limit in (lo[axis], lo[axis] + size, lo[axis] + 0.1, lo[axis] + size - 0.1, lo[axis] - 0.1):
                for off in (0.0, 1e-7, -1e-7, 1e-5, -1e-5, 1e-3, -1e-3, vs, -vs):
                    c = lo + size * rng.uniform(0.2, 0.8, 3)
                    c[axis] = limit + off
                    e = rng.normal(size=(2, 3)) * size * 0.1
                    e[:, axis] = 0.0 if rng.random() < 0.6 else rng.normal(size=2) * 1e-5
                    tris.append([c, c + e[0], c + e[1]])
    scene = _pack(np.array(tris, np.float32), rng)
    ds, ws = passes.DeviceScene(scene), passes.Workspace()
    opacity = clipmap.new_atlas(R)
    passes.voxelize_opacity(ds, regions, R, opacity, ws)
    want = oracle.voxelize_opacity(scene, R, reg)
    assert np.array_equal(opacity.cpu().numpy().view(np.uint32), want) and want.any()
