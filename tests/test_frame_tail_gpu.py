"""A deterministic frame's streaming passes over voxel bitmaps (opacity atlas from bits, radiance outside the mips'
blocks, mips that skip empty children) against the same frame pass by pass through the ABI, texel for texel: grids
from 8 to 128 (rows of fewer bits than a word, and more), frames on which some levels are due, stale atlas contents,
cameras on both sides of zero (wrapped blocks), both opacity formats, the toroidal update, unaligned atlases, and the
radiance texture the frame keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)


def _dirty(torch, R, seed, dtype, offset=0):
    """An atlas full of stale words, its first texel `offset` texels past an aligned address."""
    D, H = R + 2, 6 * (R + 2)
    g = torch.Generator(device="cuda").manual_seed(seed)
    hi = 256 if dtype == torch.uint8 else (1 << 31) - 1
    flat = torch.randint(0, hi, (D * H * H + offset,), generator=g, device="cuda", dtype=torch.int64).to(dtype)
    return flat[offset:].view(D, H, H)


def _interior(torch, R):
    """Texels that are interior in all three axes (radiance borders are never written)."""
    i = torch.arange(6 * (R + 2), device="cuda") % (R + 2)
    i = (i >= 1) & (i <= R)
    z = torch.arange(R + 2, device="cuda")
    z = (z >= 1) & (z <= R)
    return z[:, None, None] & i[None, :, None] & i[None, None, :]


def _levels(torch, R, due):
    y = torch.arange(6 * (R + 2), device="cuda") // (R + 2)
    return torch.tensor([bool((due >> l) & 1) for l in range(6)], device="cuda")[y][None, :, None]


@pytest.fixture(scope="module")
def setup(cuda):
    from vk_voxel_cone_tracing_gb300 import passes
    from vk_voxel_cone_tracing_gb300.scene import room_scene
    scene = room_scene(seed=12, n_random=2500)
    scene.materials["emissive_factor"][::11] = (0.4, 0.0, 0.9)
    return passes.DeviceScene(scene), passes.Workspace()


@pytest.mark.parametrize("R", [8, 16, 32, 128])
@pytest.mark.parametrize("index,camera", [(0, (0.4, 3.0, -0.3)), (2, (-7.3, 2.0, 5.1)), (1, (3.0, 4.0, -2.0))])
@pytest.mark.parametrize("form", ["rgba8", "r8", "unaligned", "unaligned r8"])
def test_frame_equals_its_passes(cuda, setup, R, index, camera, form):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap, passes
    ds, ws = setup
    r8, off = "r8" in form, 1 if "unaligned" in form else 0
    light = passes.light_desc(LIGHT_DIR)
    sd = passes.light_shadow_desc((-4.0, 16.0, -3.0), LIGHT_DIR)
    shadow = torch.empty((200, 256), dtype=torch.float32, device="cuda")
    radiance = _dirty(torch, R, 1, torch.int32, off)
    opacity = _dirty(torch, R, 2, torch.uint8 if r8 else torch.int32, off)
    start = radiance.clone()
    tex = clipmap.RadianceTexture(R).update(start.contiguous())
    regions = passes.clipmap_frame(ds, camera, R, opacity, radiance, shadow, light, sd, ws, frame_index=index, texture=tex,
                                   opacity_format=capi.OPACITY_R8 if r8 else capi.OPACITY_RGBA8)
    due = sum(1 << l for l in range(6) if index % (1 << l) == 0)
    # pass by pass
    o, r = clipmap.new_atlas(R), start.clone()
    passes.voxelize_opacity(ds, regions, R, o, ws)
    clipmap.cmd_downsample_all(o, R, regions, 0)
    clipmap.cmd_wrap_border(o, R)
    sh = torch.empty_like(shadow)
    passes.shadow_depth(ds, sd, sh, ws)
    for l in range(6):
        if (due >> l) & 1:
            clipmap.cmd_clear_region(r, R, (0, 0, 0), (R, R, R), l)
    passes.inject_radiance(ds, regions, R, sh, light, sd, r, ws, level_mask=due)
    for l in range(6):
        if (due >> l) & 1:
            clipmap.cmd_copy_alpha(r, o, R, l)
    for l in range(1, 6):
        if (due >> l) & 1:
            clipmap.cmd_downsample(r, R, tuple(regions[l - 1].min_corner), l, 1)
    if r8:
        assert torch.equal(opacity, (o >> 24).to(torch.uint8))
    else:
        assert torch.equal(opacity, o)
    assert torch.equal(radiance, r)
    changed = _interior(torch, R) & _levels(torch, R, due)
    assert torch.equal(torch.where(changed, 0, radiance), torch.where(changed, 0, start))
    out = torch.empty_like(r)
    tex.read(out)
    assert torch.equal(out, r)
    tex.close()


@pytest.mark.parametrize("off", [0, 1])
def test_toroidal_frame_equals_its_passes(cuda, setup, off):
    """A toroidal frame's radiance (alpha from the opacity atlas, no opacity bits) after a full one."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap, passes
    ds, ws = setup
    R, light = 32, passes.light_desc(LIGHT_DIR)
    sd = passes.light_shadow_desc((-4.0, 16.0, -3.0), LIGHT_DIR)
    shadow = torch.empty((200, 256), dtype=torch.float32, device="cuda")
    radiance, opacity = _dirty(torch, R, 1, torch.int32, off), _dirty(torch, R, 2, torch.int32, off)
    state = (capi.ClipmapRegion * 6)()
    passes.clipmap_frame(ds, (0.0, 3.0, 0.0), R, opacity, radiance, shadow, light, sd, ws, regions_state=state)
    before = radiance.clone()
    regions = passes.clipmap_frame(ds, (1.3, 3.4, -2.1), R, opacity, radiance, shadow, light, sd, ws, frame_index=4,
                                   revoxelization=capi.REVOX_TOROIDAL, regions_state=state)
    r = before.clone()
    for l in range(3):
        clipmap.cmd_clear_region(r, R, (0, 0, 0), (R, R, R), l)
    passes.inject_radiance(ds, regions, R, shadow, light, sd, r, ws, level_mask=7)
    o = opacity.clone()
    for l in range(3):
        clipmap.cmd_copy_alpha(r, o, R, l)
    for l in range(1, 3):
        clipmap.cmd_downsample(r, R, tuple(regions[l - 1].min_corner), l, 1)
    assert torch.equal(radiance, r)
