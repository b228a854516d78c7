"""A workspace that ends where a pass's needs end: the pass neither grows it nor writes behind it."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

LIGHT_DIR = (0.3, -1.0, 0.2)
PATTERN = -0x54545455


def address(ws):
    return C.cast(ws.handle, C.POINTER(C.c_void_p))[0]  # the struct begins with the arena


@pytest.mark.parametrize("mode", ["atomic", "opacity", "shadow"])
def test_nothing_is_written_behind_an_exact_workspace(cuda, mode):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap, engine, passes
    from vk_voxel_cone_tracing_gb300.scene import _pack, room_scene
    R = 16
    regions = clipmap.clip_regions((0.3, 2.0, -0.4), R)
    sd = passes.light_shadow_desc((-4.0, 16.0, -3.0), LIGHT_DIR)
    atlas = clipmap.new_atlas(R)
    depth = torch.empty((64, 64), dtype=torch.float32, device="cuda")
    adjacent = 0
    for n_random in (100, 500, 900, 1300, 1700, 2100):
        ds = passes.DeviceScene(room_scene(seed=2, n_random=n_random))

        def run(ws):
            if mode == "atomic":
                passes.inject_radiance(ds, regions, R, None, passes.light_desc(LIGHT_DIR),
                                       capi.DirectionalLightShadowDesc(), atlas, ws, mode=capi.INJECT_ATOMIC)
            elif mode == "opacity":
                passes.voxelize_opacity(ds, regions, R, atlas, ws)
            else:
                passes.shadow_depth(ds, sd, depth, ws)
            torch.cuda.synchronize()

        grown = passes.Workspace()
        run(grown)
        lo, hi = 1, grown.nbytes // 256  # the least number of 256-byte lines that is not grown
        grown.close()
        while lo < hi:
            mid = (lo + hi) // 2
            ws = passes.Workspace(256 * mid)
            run(ws)
            if ws.nbytes == 256 * mid:
                hi = mid
            else:
                lo = mid + 1
            ws.close()
        many = [passes.Workspace(256 * hi) for _ in range(16)]  # some of them side by side
        at = {address(w): w for w in many}
        for w in many:
            behind = at.get(address(w) + w.nbytes)
            if behind is None:
                continue
            adjacent += 1
            guard = engine._device_view(address(behind), (64,))
            guard.fill_(PATTERN)
            run(w)
            assert w.nbytes == 256 * hi and bool((guard == PATTERN).all())
        for w in many:
            w.close()
    if not adjacent:
        pytest.skip("no two workspaces lie side by side here")
