"""The one-kernel gradients (128-row tiles, weight gradients summed in TMEM
over a CTA's tiles) against the warp-level kernels: part of a tile, whole
tiles, one more row, and batches that give every CTA several tiles.

Both round the same numbers to BF16 and sum in FP32, so they differ by the
order of the sums, and where that moves a value over a rounding boundary by a
BF16 step of it (2^-8): well below 1e-2 of the gradient's norm."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _near(a, b):
    return np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-9


@pytest.mark.parametrize("encoding", ["hashgrid", "freq12"])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128 + 1, 3 * 148 * 128 + 77])
def test_gradients_match_the_warp_kernels(n, encoding):
    from illuminaprt_b200.ilg import GpuSpace
    sp = GpuSpace()
    sp.mlp_init(seed=4, lr=1e-2, encoding=encoding)
    raw, tgt = mo.random_batch(n, seed=21)
    want = sp.mlp_grads(raw, tgt, warp_mma=True)
    want_grid = sp.mlp_grid_grads() if encoding == "hashgrid" else None
    for _ in range(2):  # (the second call finds used scratch)
        loss, g = sp.mlp_grads(raw, tgt)
        assert abs(loss - want[0]) < 1e-2 * want[0]
        at = 0
        for rows, cols in [(96, 64)] + [(64, 64)] * 4 + [(64, 8)]:  # every layer by itself
            part = slice(at, at + rows * cols)
            assert _near(g[part], want[1][part])
            at += rows * cols
        if want_grid is not None:
            assert _near(sp.mlp_grid_grads(), want_grid)
    sp.close()
