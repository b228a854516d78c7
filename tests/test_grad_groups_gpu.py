"""The adjoint of specular cones marched by several lanes each, and of cones long enough that segments are marched
again from their checkpoints: samples repeated until one lane marches a cone (and 220 steps are 220 rounds) give the
few samples' gradient times the repeats."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("times", [150, 290, 600])  # lanes per cone: 4, 2, 1 on 608 blocks (the 256 samples alone: 8)
def test_repeated_samples_scale_the_gradient(cuda, oracle, times):
    torch = cuda
    import ctypes as C
    from vk_voxel_cone_tracing_gb300 import capi, clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_samples, smooth_volume
    R, eye = 64, (0.0, 3.0, -3.0)
    vol = torch.from_numpy(smooth_volume(R, seed=9).reshape(-1)).cuda()
    regions = oracle.clip_regions((0.2, 1.1, -0.4), R)
    desc = clipmap.trace_desc(**{**default_trace_desc(regions, R), "rendering_mode": 6})
    rec = random_samples(256, (0.2, 1.1, -0.4), 3.0, seed=10, specular_fraction=1.0)
    few = clipmap.samples_to_device(rec)
    cam, light = clipmap.cam_matrix(eye), capi.DirectionalLightDesc(capi.f3(0.3, -1.0, 0.2), 1.0, capi.f3(1, 1, 1), 0)
    weights = torch.randn((256, 4), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))

    def gradient(s, w):
        G, v = torch.zeros_like(vol), lambda t: C.c_void_p(t.data_ptr())
        capi.call("vct_cone_trace_backward", capi.ref(desc), capi.ref(cam), v(vol), R, None, capi.ref(light), None,
                  v(s), s.shape[0], v(w), v(w), v(G), None)
        return G.double()

    want = gradient(few, weights)
    got = gradient(few.repeat(times, 1), weights.repeat(times, 1)) / times
    assert (want != 0).sum() > 10000
    # a texel takes at most 2^14 shares, each rounded to 2^-24 of the sum so far
    assert float((got - want).norm() / want.norm()) < 1e-3
