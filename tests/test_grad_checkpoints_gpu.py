"""The adjoint of specular cones past the rounds whose records it keeps, so that segments are marched again from their
checkpoints, against reverse-mode differentiation of the FP64 oracle, at every number of lanes that share a cone.

A cone of s steps marched by g lanes takes s / g rounds, of which 48 are kept: the samples' longest cones take more
than 48 x 8 steps, so every run below checkpoints.  How many lanes share a cone follows from the length of the list;
it is lengthened with cones of another aperture (listed after the samples' own) that carry no weight, by factors of
two from a list that takes eight lanes to one that takes one on any grid of up to 2048 threads an SM."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R, EYE, CENTER = 32, (0.0, 3.0, -3.0), (0.2, 1.1, -0.4)
STORED_ROUNDS, MOST_LANES = 48, 8


def make_samples(n, seed):
    from vk_voxel_cone_tracing_gb300.scene import random_samples
    rec = random_samples(n, CENTER, 3.0, seed=seed, specular_fraction=0.6)
    rec["emission_texel"] = 0.0
    return rec


@pytest.fixture(scope="module")
def few(oracle):
    from vk_voxel_cone_tracing_gb300 import clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, smooth_volume
    vol = smooth_volume(R, seed=9)
    kw = {**default_trace_desc(oracle.clip_regions(CENTER, R), R), "voxel_size": 0.125}
    rec = make_samples(256, 10)
    rec["diffuse_texel"][:, 3] *= 0.5  # roughness 0.05 .. 0.45
    spec = clipmap.trace_desc(**{**kw, "rendering_mode": 6})  # the specular cone alone: a sample's steps are its cone's
    steps = np.array([oracle.cone_trace_f4(bytes(spec), EYE, vol, R, rec, begin=i, end=i + 1)[2]
                      for i in range(rec.shape[0])])
    assert (steps > STORED_ROUNDS * MOST_LANES).sum() >= 16, np.sort(steps)[-20:]
    rng = np.random.default_rng(3)
    weights = [rng.normal(size=(256, 4)).astype(np.float32) for _ in range(2)]
    reference = {}
    for mode in (6, 8):
        desc = clipmap.trace_desc(**{**kw, "rendering_mode": mode})
        reference[mode] = desc, oracle.cone_trace_grad_f4(bytes(desc), EYE, vol, R, rec, *weights)
    return vol, rec, steps, weights, reference


@pytest.mark.parametrize("mode,fill", [(6, 0)] + [(6, 5000 << k) for k in range(7)] + [(8, 0), (8, 320000)])
def test_recomputed_segments_match_the_fp64_gradient(cuda, few, mode, fill):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap
    vol, rec, steps, weights, reference = few
    desc, want = reference[mode]
    samples, w = clipmap.samples_to_device(rec), [torch.from_numpy(x).cuda() for x in weights]
    if fill:
        rest = make_samples(4096, 11)
        rest["diffuse_texel"][:, 3] = 1.0  # the widest aperture
        rest["specular_texel"][:, 3] = 0.5
        rest = clipmap.samples_to_device(rest)
        samples = torch.cat([samples, rest.repeat(-(-fill // 4096), 1)[:fill]]).contiguous()
        w = [torch.cat([x, torch.zeros((fill, 4), device="cuda")]).contiguous() for x in w]
    v, at = torch.from_numpy(vol.reshape(-1)).cuda(), lambda t: C.c_void_p(t.data_ptr())
    grad = torch.zeros_like(v)
    cam, light = clipmap.cam_matrix(EYE), capi.DirectionalLightDesc(capi.f3(0.3, -1.0, 0.2), 1.0, capi.f3(1, 1, 1), 0)
    capi.call("vct_cone_trace_backward", capi.ref(desc), capi.ref(cam), at(v), R, None, capi.ref(light), None,
              at(samples), samples.shape[0], at(w[0]), at(w[1]), at(grad), None)
    got = grad.cpu().numpy().astype(np.float64).reshape(vol.shape)
    err, scale = np.abs(got - want), float(np.abs(want).max())
    big = np.abs(want) > 1e-2 * scale
    # the bars of the adjoint's other tests (1e-4 of the norm and of the largest entry; 1e-3 of an entry above 1 % of
    # the largest, for cones of up to 220 steps), the last in proportion to the steps, each of which rounds once more
    entry = 1e-3 * max(1.0, steps.max() / 220)
    stats = np.linalg.norm(err) / np.linalg.norm(want), err.max() / scale, (err[big] / np.abs(want[big])).max()
    print(mode, fill, stats, entry)
    assert np.count_nonzero(want) > 100000
    assert stats[0] < 1e-4 and stats[1] < 1e-4 and stats[2] < entry, stats
