"""Forms of rays and meshes at the edges of the wide-node traversal: axis-parallel
and signed-zero directions, origins far outside the mesh, shifted and scaled
meshes, meshes of one and two triangles, and batch sizes around a warp, a block
and the refill of idle lanes. Closest hits are the reference test's over every
triangle (ids equal up to near ties, t and barycentrics bit for bit)."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes
from tests.parity import classify

pytestmark = pytest.mark.gpu


def _rays(form, pos, idx, n, rng):
    lo, hi = pos.min(0).astype(np.float64), pos.max(0).astype(np.float64)
    o4, d4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    at = lo + rng.random((n, 3)) * (hi - lo)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if form == "axis":
        d = np.eye(3)[rng.integers(0, 3, n)] * rng.choice([-1.0, 1.0], (n, 1))
        d = np.where(d == 0, rng.choice([-0.0, 0.0], (n, 3)), d)
        at = at - d * (hi - lo).max()
    elif form == "far":
        at = at - d * 1e3 * (hi - lo).max()
    elif form == "plane":  # one zero component
        d[np.arange(n), rng.integers(0, 3, n)] = 0.0
        at = at - d * (hi - lo).max()
    o4[:, :3], d4[:, :3], d4[:, 3] = at, d, scenes.FLT_MAX
    return o4, d4


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1025, 16385, 40961])
@pytest.mark.parametrize("form", ["axis", "far", "plane", "inside"])
@pytest.mark.parametrize("mesh", ["one", "two", "grid", "shifted", "tiny"])
def test_closest_and_any_hits_match_brute_force(mesh, form, n, oracle):
    from illuminaprt_b200.ilg import GpuSpace
    rng = np.random.default_rng([n, len(form), len(mesh)])
    if mesh in ("one", "two"):
        pos = np.array([[0, 0, 0], [1, 0, 0.1], [0, 1, 0.2], [1, 1, 0]], np.float32)
        idx = np.array([[0, 1, 2], [1, 3, 2]], np.uint32)[:1 if mesh == "one" else 2]
    else:
        pos, idx = scenes.heightfield(24, 17, 0.4, 3)
        if mesh == "shifted":
            pos = (pos * np.float32(64) + np.float32([1000, -300, 20])).astype(np.float32)
        elif mesh == "tiny":
            pos = (pos * np.float32(0.03125)).astype(np.float32)
    o4, d4 = _rays(form, pos, idx, n, rng)
    sp = GpuSpace()
    sp.initialise(pos, idx)
    sp.build()
    got = sp.intersects(o4, d4)
    ref = oracle.intersect_brute(pos, idx, o4, d4)
    n_same, ties, bad, bits_ok = classify(pos, idx, o4, d4, got, ref, oracle)
    assert bad == [] and bits_ok and ties <= 2 + n // 100
    assert np.array_equal(sp.occluded(o4, d4).astype(bool), ref[0] >= 0)
    half = idx.shape[0] // 2  # the excluding kernels: the first half left out
    if half:
        p = sp.intersects_excluding(o4, d4, 0, half)[0]
        assert np.array_equal(p >= 0, oracle.intersect_brute(pos, idx[half:], o4, d4)[0] >= 0)
    sp.close()
