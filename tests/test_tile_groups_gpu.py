"""The octree's fragment list where chunks take eight consecutive tiles (3 x 2^19 tiles and more) and four (from 2^20):
the list of a scene is the list of its first triangles followed by that of the rest."""
import copy

import pytest

pytestmark = pytest.mark.gpu


def test_long_lists_are_their_parts(cuda):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, passes
    from vk_voxel_cone_tracing_gb300.scene import terrain_scene
    scene = terrain_scene(seed=5, target=2_300_000, boxes=7000)  # a tile a triangle or more
    T, ws, sd = scene.indices.shape[0], passes.Workspace(), capi.DirectionalLightShadowDesc()
    whole = passes.DeviceScene(scene)
    lists = []
    for lo, hi in ((0, T), (0, T // 8), (T // 8, T // 2), (T // 2, T)):
        part = copy.copy(scene)
        part.indices, part.tri_material = scene.indices[lo:hi], scene.tri_material[lo:hi]
        lists.append(passes.svo_fragments(passes.DeviceScene(part), 8, None, passes.light_desc((0.3, -1.0, 0.2)), sd, ws,
                                          bb_min=whole.bb_min, bb_max=whole.bb_max))
    assert T > 2_200_000 and lists[0].shape[0] > 1 << 21
    assert torch.equal(lists[0], torch.cat(lists[1:]))
