"""Device builds at the sizes where the bottom-up passes and the eight-lane
collapse change shape: one to nine triangles, sizes around a treelet, a warp
and a block, meshes of identical and degenerate triangles, and rebuilds of
growing and shrinking meshes in one context (the scratch is kept between
builds). Closest hits are the reference test's over every triangle."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes
from tests.parity import classify

pytestmark = pytest.mark.gpu


def _check(sp, pos, idx, oracle, seed):
    sp.initialise(pos, idx)
    sp.build()
    st = sp.stats()
    assert st["n_leaf_tris"] == idx.shape[0] and 1 <= st["n_nodes"] <= idx.shape[0]
    rng = np.random.default_rng(seed)
    lo, hi = pos.min(0).astype(np.float64), pos.max(0).astype(np.float64)
    n = 700
    o4, d4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o4[:, :3] = lo + rng.random((n, 3)) * (hi - lo) - 2.0 * d
    d4[:, :3], d4[:, 3] = d, scenes.FLT_MAX
    got, ref = sp.intersects(o4, d4), oracle.intersect_brute(pos, idx, o4, d4)
    n_same, ties, bad, bits_ok = classify(pos, idx, o4, d4, got, ref, oracle)
    assert bad == [] and bits_ok


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 6, 7, 8, 9, 31, 32, 33, 63, 129, 512, 513, 4097])
def test_small_and_odd_meshes(n, fast, oracle):
    from illuminaprt_b200.ilg import GpuSpace
    pos, idx = scenes.heightfield(64, 33, 0.4, 5)
    sp = GpuSpace(fast_build=fast)
    _check(sp, pos, np.random.default_rng(n).permutation(idx)[:n], oracle, n)
    sp.close()


def test_identical_and_degenerate_triangles(oracle):
    from illuminaprt_b200.ilg import GpuSpace
    pos, idx = scenes.heightfield(8, 4, 0.4, 5)
    sp = GpuSpace()
    same = np.repeat(idx[:1], 100, 0)
    points = np.repeat(idx[:, :1], 3, 1)  # every vertex the same: no area, no hits
    _check(sp, pos, np.concatenate([same, points, idx]), oracle, 1)
    sp.close()


def test_rebuilds_in_one_context(oracle):
    from illuminaprt_b200.ilg import GpuSpace
    sp = GpuSpace()
    for k, (nx, ny) in enumerate([(5, 3), (90, 41), (2, 1), (200, 60), (90, 41)]):
        pos, idx = scenes.heightfield(nx, ny, 0.3, k)
        _check(sp, pos, idx, oracle, k)
        sp.build()  # again on the same mesh
        _check(sp, pos, idx, oracle, k)
    sp.close()
