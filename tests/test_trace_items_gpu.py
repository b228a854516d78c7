"""Traces of few samples give each warp item fewer of them (deal_samples_per_warp) and list their specular cones by
blocks of 1024: a sample's outputs do not depend on how many others are traced with it, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cones32", [0, 1])
def test_rows_equal_in_traces_of_every_size(cuda, oracle, cones32):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_atlas, random_samples
    R, n = 32, 180000
    regions = oracle.clip_regions((0.0, 0.0, 0.0), R)
    atlas = torch.from_numpy(random_atlas(R, seed=2, fill=0.1).view(np.int32).copy()).cuda()
    tex = clipmap.RadianceTexture(R).update(atlas)
    desc = clipmap.trace_desc(**{**default_trace_desc(regions, R), "enable_32_cones": cones32})
    samples = clipmap.samples_to_device(random_samples(n, (0, 0, 0), 5.0, seed=3))
    eye = (0.0, 1.0, -4.0)
    forms = (lambda s: clipmap.cone_trace_fast(desc, eye, tex, s), lambda s: clipmap.cone_trace(desc, eye, atlas, R, s))
    for form in forms:
        want = form(samples)
        for lo, m in ((0, 1), (7, 3), (100, 33), (50, 1024), (3000, 1025), (9000, 6200), (20000, 13000), (0, 60001)):
            got = form(samples[lo:lo + m].contiguous())
            for g, w in zip(got, want):
                assert torch.equal(g, w[lo:lo + m]), (lo, m)
    tex.close()
