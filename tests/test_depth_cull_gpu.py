"""Triangles wholly outside the depth clip in the one-sample passes, which share the set-up that culls them: the
shadow depth and the G-buffer of triangles on both sides of the near and far limits, from an ulp to a unit away, flat
and tilted across, equal the oracle's word for word; and G-buffer triangles whose edge values pass 32 bits."""
import numpy as np
import pytest

from .test_gbuffer_gpu import _compare, _run

pytestmark = pytest.mark.gpu

OFFSETS = (0.0, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5, 1e-3, -1e-3, 0.05, -0.05, 1.0, -1.0)


@pytest.fixture(scope="module")
def ws(cuda):
    from vk_voxel_cone_tracing_gb300.passes import Workspace
    return Workspace()


def about_planes(rng, origin, direction, distances, spread, per):
    """Triangles at `distances` (and OFFSETS from them) along `direction`, flat across it or tilted."""
    d = np.asarray(direction, np.float64)
    d /= np.linalg.norm(d)
    side = np.cross(d, (0.0, 1.0, 0.1))
    side /= np.linalg.norm(side)
    up = np.cross(side, d)
    tris = []
    for t in distances:
        for off in OFFSETS:
            for k in range(per):
                c = np.asarray(origin) + d * (t + off) + (side * rng.uniform(-1, 1) + up * rng.uniform(-1, 1)) * spread(t)
                e = [(side * rng.normal() + up * rng.normal()) * 0.3 * spread(t) + d * tilt
                     for tilt in rng.normal(size=2) * rng.choice([0.0, 1e-6, 1e-2])]
                tris.append([c, c + e[0], c + e[1]])
    return np.array(tris, np.float32)


@pytest.mark.parametrize("width,height", [(512, 512), (333, 257)])
def test_shadow_depth_about_the_limits(cuda, oracle, ws, width, height):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import passes
    from vk_voxel_cone_tracing_gb300.scene import _pack
    rng = np.random.default_rng(width)
    origin, direction = (-4.0, 16.0, -3.0), (0.3, -1.0, 0.2)
    scene = _pack(about_planes(rng, origin, direction, (0.1, 30.0), lambda t: 12.0, 8), rng)
    depth = torch.empty((height, width), dtype=torch.float32, device="cuda")
    passes.shadow_depth(passes.DeviceScene(scene), passes.light_shadow_desc(origin, direction), depth, ws)
    want = oracle.shadow_depth(scene, oracle.light_shadow_desc(origin, direction), width, height)
    got = depth.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), np.count_nonzero(got != want)
    assert (want < 0.5).any() and ((want > 0.5) & (want < 1.0)).any()  # some at either limit are inside


def test_gbuffer_about_the_limits(cuda, oracle, ws):
    from vk_voxel_cone_tracing_gb300.scene import _pack
    rng = np.random.default_rng(5)
    pos, direction, W, H = (0.3, 2.0, -4.0), (0.2, -0.1, 1.0), 203, 117
    cam = oracle.camera_matrix(pos, direction, aspect=W / H)
    # the camera's limits are 0.01 and 5000; depths pass 1 + 2^-20, from which on all are culled, near 9600
    distances = (0.01, 4900.0, 5000.0, 5100.0, 9600.0, 30000.0)
    scene = _pack(about_planes(rng, pos, direction, distances, lambda t: 0.4 * t, 12), rng)
    want = oracle.gbuffer(scene, cam, W, H)
    got = _run(cuda, scene, cam, W, H, ws)
    assert (want[:, 3] < 1.0).any()
    _compare(got, want)


@pytest.mark.parametrize("W,H", [(1280, 720), (1531, 900)])
def test_gbuffer_triangles_past_32_bit_edges(cuda, oracle, ws, W, H):
    """Edges longer than 512 pixels (deltas of 2^17 1/256 pixels) and edge values past 2^31, fanned with shared edges
    and small triangles before them."""
    from vk_voxel_cone_tracing_gb300.scene import _pack
    rng = np.random.default_rng(W)
    tris = []
    for size in (0.3, 1.5, 2.9, 3.1, 6.0, 20.0, 90.0):
        c = np.array([0.0, 2.0, 3.0]) + rng.uniform(-1, 1, 3) * (0.5, 0.5, 2.0)
        e = rng.normal(size=(2, 3)) * (1.0, 1.0, 0.2)
        e = e / np.linalg.norm(e, axis=1, keepdims=True) * size
        a, b = c + e[0], c + e[1]
        tris += [[c, a, a + e[1]], [c, a + e[1], b], [c, b, c - e[0]]]
    scene = _pack(np.array(tris, np.float32), rng)
    cam = oracle.camera_matrix((0.0, 2.0, 0.0), (0.05, 0.02, 1.0), aspect=W / H)
    want = oracle.gbuffer(scene, cam, W, H)
    _compare(_run(cuda, scene, cam, W, H, ws), want)
    assert (want[:, 3] < 1.0).mean() > 0.5
