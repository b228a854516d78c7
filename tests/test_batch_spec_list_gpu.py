"""The specular list of a batched trace on both sides of the size from which it is made in order: every job's outputs
and step count equal those of the job traced alone, with jobs of no, one and all specular samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 1 << 18  # 32-padded positions


@pytest.mark.parametrize("positions", [LIMIT - 32, LIMIT, LIMIT + 4128])
@pytest.mark.parametrize("specular", [(0.5, 0.0, 1.0), (0.0, 0.0, 0.0)])
def test_batch_equals_each_job_alone(cuda, positions, specular):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_atlas, random_samples
    R = 16
    sizes = [1, 33, 70001]
    rest = positions - sum((n + 31) // 32 * 32 for n in sizes)
    sizes.append(rest - 31)  # one sample in its last 32 positions
    records, want, got = [], [], []
    for k, n in enumerate(sizes):
        regions = clipmap.clip_regions((0.3 * k, 0.0, 0.1 * k), R)
        desc = clipmap.trace_desc(**default_trace_desc(clipmap.regions_to_numpy(regions), R))
        atlas = random_atlas(R, seed=k, fill=0.1)
        tex = clipmap.RadianceTexture(R).update(torch.from_numpy(atlas.view(np.int32).copy()).cuda())
        rec = random_samples(n, (0, 0, 0), 3.0, seed=20 + k, specular_fraction=specular[k % 3])
        rec["specular_texel"][-1, 3] = max(specular)  # the last position's
        dev, eye = clipmap.samples_to_device(rec), (0.5, 1.0, -4.0)
        st = [torch.zeros(1, dtype=torch.int64, device="cuda") for _ in range(2)]
        want.append((*clipmap.cone_trace_fast(desc, eye, tex, dev, steps=st[0]), st[0]))
        got.append((torch.full((n, 4), -3.0, device="cuda"), torch.full((n, 4), -3.0, device="cuda"), st[1]))
        records.append((clipmap.trace_job(desc, eye, tex, dev, *got[-1][:2], steps=st[1]), tex, dev))
    clipmap.cone_trace_fast_batch([r[0] for r in records])
    torch.cuda.synchronize()
    for k, (g, w) in enumerate(zip(got, want)):
        assert all(torch.equal(a, b) for a, b in zip(g, w)), k
    lit = [float(w[1][:, :3].abs().sum()) > 0 for w in want]
    assert any(lit) == (max(specular) > 0)
