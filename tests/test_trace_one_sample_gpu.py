"""The per-sample traces of a single sample captured in a CUDA graph: a replay reads the sample as it is then, and
nothing of the host frame that captured it."""
import pytest

pytestmark = pytest.mark.gpu

BOX = dict(bb_min=(-4.0, -4.0, -4.0), bb_max=(4.0, 4.0, 4.0))


@pytest.mark.parametrize("form", ["octree", "exact", "texels"])
@pytest.mark.parametrize("n", [1, 2])
def test_captured_trace_replays(cuda, form, n):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_atlas, random_samples

    from .test_svo_trace_rules import dense_pool
    R, eye = 32, (0.0, 1.0, -4.0)
    regions = clipmap.clip_regions((0.0, 0.0, 0.0), R)
    desc = clipmap.trace_desc(**default_trace_desc(clipmap.regions_to_numpy(regions), R))
    samples = clipmap.samples_to_device(random_samples(2 * n, (0, 0, 0), 3.0, seed=5, specular_fraction=1.0))
    if form == "octree":
        pool = torch.from_numpy(dense_pool(5, 3).view("i4").copy()).cuda()
        trace = lambda s: passes.svo_cone_trace(desc, eye, pool, pool.shape[0], s, **BOX)
    else:
        atlas = torch.from_numpy(random_atlas(R, seed=1, fill=0.3).view("i4").copy()).cuda()
        if form == "texels":
            tex = clipmap.RadianceTexture(R).update(atlas)
            trace = lambda s: clipmap.cone_trace_tex(desc, eye, tex, s)
        else:
            trace = lambda s: clipmap.cone_trace(desc, eye, atlas, R, s)
    want = [[t.clone() for t in trace(samples[k * n:(k + 1) * n].contiguous())] for k in (0, 1)]
    assert not torch.equal(want[0][0], want[1][0]) and float(want[0][1][:, :3].abs().sum()) > 0
    given = samples[:n].clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = trace(given)
    for k in (0, 1, 0):
        given.copy_(samples[k * n:(k + 1) * n])
        graph.replay()
        torch.cuda.synchronize()
        for got, w in zip(out, want[k]):
            assert torch.equal(got, w), k
