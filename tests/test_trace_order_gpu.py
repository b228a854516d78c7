"""The fast trace's visiting order on both sides of the sample count (by clipmap resolution) from which it is sorted by
the keys' low bits too, with and without the high ones: the outputs and step counts are those of the same samples
traced in pieces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [8, 32, 256])
@pytest.mark.parametrize("over", [-1, 0, 1])
def test_order_does_not_change_a_sample(cuda, R, over):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_atlas, random_samples
    n = (2048 if R <= 128 else 3072) * R + over
    regions = clipmap.clip_regions((0.1, 0.0, -0.2), R)
    desc = clipmap.trace_desc(**default_trace_desc(clipmap.regions_to_numpy(regions), R))
    tex = clipmap.RadianceTexture(R).update(torch.from_numpy(random_atlas(R, seed=4, fill=0.1).view(np.int32).copy()).cuda())
    samples, eye = clipmap.samples_to_device(random_samples(n, (0, 0, 0), 30.0, seed=R)), (0.5, 1.0, -4.0)

    def trace(s):
        steps = torch.zeros(1, dtype=torch.int64, device="cuda")
        d, sp = clipmap.cone_trace_fast(desc, eye, tex, s, steps=steps)
        return d, sp, int(steps.item())

    d, sp, steps = trace(samples)
    parts = [trace(p.contiguous()) for p in samples.split(n // 3 + 1)]
    assert torch.equal(d, torch.cat([p[0] for p in parts])) and torch.equal(sp, torch.cat([p[1] for p in parts]))
    assert steps == sum(p[2] for p in parts) and float(sp[:, :3].abs().sum()) > 0
