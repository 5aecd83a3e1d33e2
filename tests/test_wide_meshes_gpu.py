"""Axis-parallel rays over meshes up to 1e18 units wide: a flat grid of 8 x 8
squares seen straight down, where the reciprocal of a zero direction component
times a node's quantisation step is the largest number of the box test. Every
ray goes through the inside of one known triangle, so the hit is known; t is
the eye's height."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = 8


@pytest.mark.parametrize("n", [200, 50000])
@pytest.mark.parametrize("watertight", [False, True])
@pytest.mark.parametrize("width", [1.0, 1e12, 1e15, 3e16, 1e17, 1e18])
def test_vertical_rays_find_their_triangle(width, watertight, n):
    from illuminaprt_b200.ilg import GpuSpace
    k = np.arange(CELLS + 1)
    x, y = np.meshgrid(k, k, indexing="ij")
    pos = np.stack([x / CELLS * width, y / CELLS * width, 0 * x], -1).reshape(-1, 3).astype(np.float32)
    a = ((x * (CELLS + 1) + y)[:-1, :-1]).reshape(-1)
    idx = np.stack([np.stack([a, a + CELLS + 1, a + CELLS + 2], -1),
                    np.stack([a, a + CELLS + 2, a + 1], -1)], 1).reshape(-1, 3).astype(np.uint32)
    tri = np.arange(n) % idx.shape[0]
    o4, d4 = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    o4[:, :3] = pos[idx[tri]].astype(np.float64).mean(1)
    o4[:, 2] = 10.0
    d4[:, 2], d4[:, 3] = -1.0, np.finfo(np.float32).max
    d4[::2, 0] = -0.0
    sp = GpuSpace()
    sp.initialise(pos, idx)
    sp.build()
    prim, t, _, _ = sp.intersects(o4, d4, watertight=watertight)
    assert np.array_equal(prim, tri) and np.allclose(t, 10.0, rtol=1e-5)
    assert sp.occluded(o4, d4, watertight=watertight).all()
    sp.close()
