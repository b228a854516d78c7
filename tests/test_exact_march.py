"""The exact trace's arithmetic short cuts and its grouped specular march.

The two-term divisions by a known divisor and the packed byte decode equal the correctly rounded quotients over
every significand and byte; a specular cone's result does not depend on how many lanes march it."""
from fractions import Fraction as F

import numpy as np
import pytest


@pytest.mark.parametrize("y", [6] + [2 + 2 ** k for k in range(12)])
def test_known_divisor_quotients_are_correctly_rounded(y):
    hi = np.float32(1.0 / y)
    lo = np.float32(1.0 / y - float(hi))
    for start in range(0, 1 << 23, 1 << 21):
        x = (np.arange(start, start + (1 << 21), dtype=np.uint32) | np.uint32(0x3F800000)).view(np.float32)
        want = x / np.float32(y)
        p, q = x.astype(np.float64) * float(hi), (x * lo).astype(np.float64)  # the product is exact (48 bits)
        s = p + q
        err = (p - s) + q  # |p| > |q|: p + q = s + err exactly
        half = np.minimum(np.spacing(want), want - np.nextafter(want, np.float32(0))).astype(np.float64) / 2
        # strictly inside half an ulp of the quotient, the fused multiply-add rounds to it
        assert (np.abs((s - want.astype(np.float64)) + err) < half).all()


def test_packed_byte_decode_is_correctly_rounded():
    for b in range(256):
        x = np.uint32(65793 * b).view(np.float32)  # the byte three times over: 65793 b 2^-149
        exact = F(float(x)) * F(2) ** 125 + F(float(x)) * F(2) ** 101
        want = np.float32(b) / np.float32(255)
        if b == 0:
            assert exact == 0
            continue
        half = min(np.spacing(want), want - np.nextafter(want, np.float32(0)))
        assert abs(exact - F(float(want))) < F(float(half)) / 2


@pytest.mark.gpu
@pytest.mark.parametrize("over", [{}, {"voxel_size": 0.3, "volume_dimension": 37.5}, {"enable_32_cones": 1}])
def test_groups_of_every_size_march_alike(cuda, oracle, over):
    """513 samples with a specular cone each, alone (8 lanes a cone) and repeated until 4, 2 and 1 lanes march one;
    the step counts too, and both reads (linear atlas and texture)."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap
    from vk_voxel_cone_tracing_gb300.scene import default_trace_desc, random_atlas, random_samples
    R = 16
    regions = oracle.clip_regions((0.0, 0.0, 0.0), R)
    atlas = torch.from_numpy(random_atlas(R, seed=4, fill=0.3).view(np.int32).copy()).cuda()
    desc = clipmap.trace_desc(**{**default_trace_desc(regions, R), "occlusion_decay": 0.05, **over})
    rec = random_samples(4000, (0, 0, 0), 4.0, seed=5)
    probe = clipmap.samples_to_device(rec)
    sout = torch.zeros((4000, 4), dtype=torch.float32, device="cuda")
    clipmap.cone_trace(desc, (0.0, 1.0, -4.0), atlas, R, probe, specular=sout)
    few = probe[sout[:, :3].abs().sum(1) > 0][:513].contiguous()
    assert few.shape[0] == 513

    def run(s):
        steps = torch.zeros(1, dtype=torch.int64, device="cuda")
        d, sp = clipmap.cone_trace(desc, (0.0, 1.0, -4.0), atlas, R, s, steps=steps)
        return d, sp, int(steps.item())

    d, sp, steps = run(few)
    for times in (60, 120, 200, 320):  # 30,780 to 164,160 cones for 155,648 lanes
        D, S, n = run(few.repeat(times, 1))
        assert torch.equal(D, d.repeat(times, 1)) and torch.equal(S, sp.repeat(times, 1))
        assert n == steps * times
    if "voxel_size" not in over:
        tex = clipmap.RadianceTexture(R).update(atlas)
        for got, want in zip(clipmap.cone_trace_tex(desc, (0.0, 1.0, -4.0), tex, few), (d, sp)):
            assert torch.equal(got, want)
        tex.close()
