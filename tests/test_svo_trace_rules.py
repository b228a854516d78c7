"""The octree trace's per-step shortcuts: cells by a multiply-add and levels by an exponent equal the shader's
expressions (CPU, float32 restated in numpy), and whole traces follow the oracle's FP32 mirror over pools that fill
the box, at voxel sizes, boxes and step factors off the usual powers of two (GPU)."""
import numpy as np
import pytest

f32 = np.float32


def cells_shader(p, c, ev, dim):
    s = (p - c) / ev
    u = ((s + f32(1.0)) * f32(0.5)) * f32(dim)
    return np.minimum(np.clip(u.astype(np.float64), 0.0, 4294967040.0).astype(np.int64), dim - 1)


@pytest.mark.parametrize("dim", [2, 64, 256, 512, 4096])
@pytest.mark.parametrize("lo,hi", [(-15.367, 14.399), (0.25, 0.26), (1000.0, 1024.0), (-3e5, 7e4)])
def test_cell_by_multiply_add(dim, lo, hi):
    c, ev = f32((f32(lo) + f32(hi)) * f32(0.5)), f32((f32(hi) - f32(lo)) * f32(0.5))
    scale = 0.5 * dim / float(ev)
    off = 0.5 * dim - float(c) * scale
    a, b = f32(scale), f32(off)
    ga, g0 = f32(abs(scale) * 2.0 ** -20), f32((abs(float(c) * scale) + dim) * 2.0 ** -20)
    rng = np.random.default_rng(dim)
    borders = (np.arange(dim + 1) / dim * 2 - 1) * float(ev) + float(c)
    p = np.concatenate([rng.uniform(lo - (hi - lo), hi + (hi - lo), 200000),
                        borders, np.repeat(borders, 8) * (1 + rng.normal(0, 1e-6, 8 * (dim + 1)))]).astype(f32)
    p = np.concatenate([p, np.nextafter(p, f32(np.inf)), np.nextafter(p, f32(-np.inf))])
    # the fused multiply-add: the product is exact in double; its sum is rounded once more, which the bound covers
    q = (p.astype(np.float64) * float(a) + float(b)).astype(f32)
    g = (np.abs(p).astype(np.float64) * float(ga) + float(g0)).astype(f32)
    r = q - np.floor(q)
    quick = (r > g) & (r < f32(1.0) - g)
    got = np.minimum(np.clip(np.floor(q).astype(np.float64), 0.0, 4294967040.0).astype(np.int64), dim - 1)
    want = cells_shader(p, c, ev, dim)
    assert np.array_equal(got[quick], want[quick])


@pytest.mark.parametrize("radius", [8.0, 0.5, 3.7, 1e-6, 12345.0])
def test_min_level_by_exponent(radius):
    radius = f32(radius)
    inv = f32(1.0 / (float(radius) * float(radius)))
    rng = np.random.default_rng(3)
    near = np.concatenate([2.0 ** k * (1 + np.arange(-400, 401) * 2.0 ** -24) for k in range(-20, 21)])
    x = np.concatenate([2.0 ** rng.uniform(-30, 30, 200000), near])
    d2 = ((x * float(radius)) ** 2).astype(f32)
    bits = (d2 * inv).astype(f32).view(np.uint32)
    rel = (bits - np.uint32(0x3f800000)).astype(np.uint32)
    slow = ((rel + np.uint32(128)) & np.uint32(0xffffff)) < 256
    slow |= (bits - np.uint32(0x0d800000)).astype(np.uint32) >= 0x64800000
    got = (rel.view(np.int32) >> 24) + 1
    ratio = (np.sqrt(d2) / radius).astype(f32)
    # any float32 logarithm within two ulp of the true one has the same ceil away from the slow cases
    true = np.log2(ratio.astype(np.float64))
    ulp = np.spacing(np.maximum(np.abs(true), 1e-30).astype(f32)).astype(np.float64)
    for t in (true, true - 2 * ulp, true + 2 * ulp):
        assert np.array_equal(got[~slow], np.ceil(t)[~slow].astype(int))


def dense_pool(depth, seed, fill=0.7):
    """A breadth-first pool over the whole box: every node of a level has children with probability `fill`."""
    rng = np.random.default_rng(seed)
    nodes, begin, num = [np.zeros((8, 2), np.uint32)], 0, 8
    pool = np.zeros((8, 2), np.uint32)
    for d in range(1, depth):
        parents = begin + np.flatnonzero(rng.random(num) < fill)
        pool[parents, 0] = (0x80000000 | (pool.shape[0] + 8 * np.arange(parents.size))).astype(np.uint32)
        begin, num = pool.shape[0], 8 * parents.size
        pool = np.concatenate([pool, np.zeros((num, 2), np.uint32)])
    words = rng.integers(0, 1 << 32, pool.shape[0], dtype=np.uint64).astype(np.uint32)
    alpha = np.minimum(rng.integers(0, 120, pool.shape[0]), 90).astype(np.uint32)
    pool[:, 1] = np.where(rng.random(pool.shape[0]) < 0.5, (words & 0xffffff) | (alpha << 24), 0)
    return pool


@pytest.mark.gpu
@pytest.mark.parametrize("dim,voxel,box,over", [
    (256, 0.0625, ((-8, -6, -8), (8, 9, 8)), {}),
    (64, 0.21, ((-4, -2, -9), (5, 3.3, 2)), dict(enable_32_cones=1)),
    (512, 0.03, ((-8, -8, -8), (8, 8, 8)), dict(min_trace_step_factor=0.1, rendering_mode=6)),
    (16, 1.5, ((-20, -20, -20), (20, 20, 20)), dict(rendering_mode=5, trace_start_offset=0.3)),
])
def test_dense_pool_against_the_oracle(cuda, oracle, dim, voxel, box, over):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import random_samples
    pool_np = dense_pool(min(6, int(np.log2(dim))), dim)
    kw = dict(volume_center=(0.4, 0.1, -0.3), rendering_mode=8, voxel_size=voxel, volume_dimension=float(dim),
              trace_start_offset=1.0, indirect_diffuse_intensity=4.0, ambient_occlusion_factor=0.5,
              min_trace_step_factor=1.0, indirect_specular_intensity=3.0, occlusion_decay=2.0, enable_32_cones=0)
    desc = clipmap.trace_desc(**{**kw, **over})
    samples = random_samples(700, (0.0, 0.5, 0.0), 5.0, seed=8)
    samples["depth"][::50] = 1.0
    eye = (0.0, 3.0, -4.0)
    d32, s32, st32 = oracle.svo_trace(32, bytes(desc), eye, pool_np, samples, *box)
    pool = torch.from_numpy(pool_np.view(np.int32).copy()).cuda()
    steps = torch.zeros(1, dtype=torch.int64, device="cuda")
    d, s = passes.svo_cone_trace(desc, eye, pool, pool_np.shape[0], clipmap.samples_to_device(samples), *box, steps=steps)
    for got, want in ((d.cpu().numpy(), d32), (s.cpu().numpy(), s32)):
        err = np.abs(got - want).max(1) / np.maximum(np.abs(want).max(1), 1e-3)
        # the mirror's bar (the host's log2 / pow / exp2 differ from the device's by an ulp; a step at a level or
        # cell border may then take its neighbour)
        assert np.mean(err < 1e-4) > 0.99, np.sort(err)[-8:]
    assert abs(int(steps.item()) - st32) <= max(8, 0.002 * st32)


@pytest.mark.gpu
def test_octree_cone_groups_march_alike(cuda):
    """The octree trace of 300 specular samples, alone (8 lanes a cone) and repeated until fewer march one."""
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import clipmap, passes
    from vk_voxel_cone_tracing_gb300.scene import random_samples
    pool = torch.from_numpy(dense_pool(5, 3).view(np.int32).copy()).cuda()
    desc = clipmap.trace_desc(volume_center=[0.0, 0.0, 0.0], rendering_mode=8, voxel_size=0.25, volume_dimension=32.0,
                              trace_start_offset=1.0, indirect_diffuse_intensity=8.0, ambient_occlusion_factor=0.5,
                              min_trace_step_factor=1.0, indirect_specular_intensity=3.0, occlusion_decay=0.05,
                              enable_32_cones=0)
    box = dict(bb_min=(-4.0, -4.0, -4.0), bb_max=(4.0, 4.0, 4.0))

    def run(s):
        steps = torch.zeros(1, dtype=torch.int64, device="cuda")
        d, sp = passes.svo_cone_trace(desc, (0.0, 1.0, -4.0), pool, pool.shape[0], s, steps=steps, **box)
        return d, sp, int(steps.item())

    probe = clipmap.samples_to_device(random_samples(3000, (0, 0, 0), 3.0, seed=6))
    few = probe[run(probe)[1][:, :3].abs().sum(1) > 0][:300].contiguous()
    assert few.shape[0] == 300
    d, sp, steps = run(few)
    for times in (150, 400, 1100):  # 45,000 to 330,000 cones for 311,296 lanes
        D, S, n = run(few.repeat(times, 1))
        assert torch.equal(torch.nan_to_num(D), torch.nan_to_num(d.repeat(times, 1)))
        assert torch.equal(S, sp.repeat(times, 1)) and n == steps * times
