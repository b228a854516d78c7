"""Arguments of a frame that are refused on the host before any device work (no GPU needed)."""
import ctypes as C

import pytest

from vk_voxel_cone_tracing_gb300 import capi


@pytest.mark.parametrize("mode", [capi.INJECT_DETERMINISTIC, capi.INJECT_ATOMIC])
@pytest.mark.parametrize("fmt", [capi.OPACITY_RGBA8, capi.OPACITY_R8])
@pytest.mark.parametrize("revox", [capi.REVOX_FULL, capi.REVOX_TOROIDAL])
def test_one_atlas_for_radiance_and_opacity_is_refused(vct_lib, mode, fmt, revox):
    f = capi.FrameDesc()
    f.clipmap_resolution, f.inject_mode, f.opacity_format, f.revoxelization = 16, mode, fmt, revox
    state = (capi.ClipmapRegion * 6)()
    f.regions_state = C.cast(state, C.c_void_p)
    workspace = C.create_string_buffer(512)  # an empty one
    with pytest.raises(capi.VctError, match="must differ") as e:
        capi.call("vct_clipmap_frame", capi.ref(capi.Scene()), capi.ref(f), C.c_void_p(256), C.c_void_p(256), None, None,
                  C.cast(workspace, C.c_void_p), None)
    assert e.value.code == capi.VCT_E_BAD_ARG
    assert bytes(state) == bytes(len(bytes(state)))  # the caller's regions are left as they were
