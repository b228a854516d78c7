"""The sorted build of the octree pool (runs of equal positions, sorted by path) against the oracle's level-by-level
build, word for word, at every depth from 1 to 11 (the 33-bit path takes 64-bit keys), for lists whose positions
repeat in runs, in no order, or all at once, with any colour word (alpha wraps, zero words of discarded fragments) and
leaves long enough for the warp's fold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fragments(level, kind, n, seed):
    rng = np.random.default_rng(seed)
    res = 1 << level
    if kind == "scattered":
        p = rng.integers(0, res + 1, (n, 3))
    elif kind == "runs":  # a walk: neighbours mostly share their voxel, and come back to it later
        p = np.clip(np.cumsum(rng.integers(-1, 2, (n, 3)) * (rng.random((n, 1)) < 0.15), 0) + res // 3, 0, res)
    else:  # a few voxels hold almost everything
        p = rng.integers(0, res + 1, (4, 3))[rng.integers(0, 4, n)]
        p[rng.random(n) < 0.01] = rng.integers(0, res + 1, 3)
    p = np.minimum(p, 4095).astype(np.uint32)
    word = rng.integers(0, 1 << 28, n, dtype=np.uint32)
    if kind != "scattered":
        word = np.where(rng.random(n) < 0.5, (word & 0xffffff) | (15 << 24), word).astype(np.uint32)
    f = np.zeros((n, 2), np.uint32)
    f[:, 0] = p[:, 0] | (p[:, 1] << 12) | ((p[:, 2] & 0xff) << 24)
    f[:, 1] = ((p[:, 2] >> 8) << 28) | word
    f[rng.random(n) < (0.3 if kind == "piled" else 0.05)] = 0
    return f


@pytest.mark.parametrize("level", [1, 2, 3, 5, 8, 10, 11])
@pytest.mark.parametrize("kind,n", [("scattered", 1), ("scattered", 257), ("scattered", 30000), ("runs", 70000),
                                    ("piled", 40000)])
def test_build_equals_the_oracle(cuda, oracle, level, kind, n):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, passes
    f = fragments(level, kind, n, 100 * level + n)
    want, n_want = oracle.svo_build(f, level, capacity=4_000_000)
    ws = passes.Workspace()
    pool, nodes = passes.svo_build(torch.from_numpy(f.view(np.int32)).cuda(), level, ws, capacity=4_000_000)
    assert nodes == n_want
    got = pool[:nodes].cpu().numpy().view(np.uint32)
    assert np.array_equal(got, want[:nodes]), np.flatnonzero((got != want[:nodes]).any(1))[:8]
    if nodes > 8:
        with pytest.raises(capi.VctError) as e:
            passes.svo_build(torch.from_numpy(f.view(np.int32)).cuda(), level, ws, capacity=nodes - 1)
        assert e.value.code == capi.VCT_E_OVERFLOW
    ws.close()


def test_build_of_an_empty_list(cuda):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import passes
    pool, nodes = passes.svo_build(torch.empty((0, 2), dtype=torch.int32, device="cuda"), 6, passes.Workspace())
    assert nodes == 8 and not pool[:8].any().item()
