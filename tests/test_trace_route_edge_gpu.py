"""Both sides of the line between the eight-lanes-a-ray kernel (batches of at
most 40,960 rays) and the persistent one: the same rays, one more in the batch.
Closest and any hits with either triangle test, from host arrays (staged above
16,384 rays) and from device arrays.

The two meet triangles in one order with one arithmetic, so where they name the
same triangle t, u and v are equal bit for bit; of two hits less than the
window's 1e-5 apart either may win, as between any two traversals. What an
any-hit query answers does not depend on the order at all."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu

LINE = 40960
TIE = 1e-5


def _same_hits(a, b):
    same = a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(x[same].view(np.uint32), y[same].view(np.uint32))
    off = ~same
    assert (a[0][off] >= 0).all() and (b[0][off] >= 0).all()
    assert (np.abs(a[1][off].astype(np.float64) - b[1][off]) < TIE).all()
    assert off.sum() <= 2 + same.size // 1000


@pytest.mark.parametrize("kind", ["incoherent", "coherent"])
@pytest.mark.parametrize("watertight", [False, True])
def test_small_and_persistent_kernels_agree(watertight, kind):
    import torch
    from illuminaprt_b200.ilg import GpuSpace
    pos, idx = scenes.heightfield(220, 97, 0.3, 5)
    if kind == "coherent":
        o4, d4 = scenes.pinhole_rays(256, 161, (0.45, -0.6, 0.75), (0.5, 0.5, 0.0), (0, 0, 1), 60.0)
        o4, d4 = o4[:LINE + 1], d4[:LINE + 1]
    else:
        o4, d4 = scenes.incoherent_rays(pos, idx, LINE + 1, seed=8)
    o4, d4 = np.ascontiguousarray(o4, np.float32), np.ascontiguousarray(d4, np.float32)
    assert o4.shape[0] == LINE + 1
    sp = GpuSpace()
    sp.initialise(pos, idx)
    sp.build()
    want = sp.intersects(o4, d4, watertight=watertight)
    want_occ = sp.occluded(o4, d4, watertight=watertight)
    assert np.array_equal(want_occ.astype(bool), want[0] >= 0) and 0.1 < want_occ.mean()
    do, dd = torch.from_numpy(o4).cuda(), torch.from_numpy(d4).cuda()
    hit = [torch.empty(LINE, dtype=torch.int32, device="cuda")] + \
          [torch.empty(LINE, dtype=torch.float32, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    for n in (LINE, 16385, 16384, 7):
        part = [w[:n] for w in want]
        _same_hits(sp.intersects(o4[:n], d4[:n], watertight=watertight), part)
        assert np.array_equal(sp.occluded(o4[:n], d4[:n], watertight=watertight), want_occ[:n])
        out = [h[:n] for h in hit]
        sp.intersects_into(do[:n], dd[:n], *out, device_ptrs=True, watertight=watertight)
        sp.sync()
        _same_hits([h.cpu().numpy() for h in out], part)
    if not watertight:
        occ = torch.empty(LINE, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        sp.occluded_into(do[:LINE], dd[:LINE], occ, device_ptrs=True)
        sp.sync()
        assert np.array_equal(occ.cpu().numpy(), want_occ[:LINE])
    sp.close()
