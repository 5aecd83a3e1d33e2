"""A frame's captured launches are replayed only for the light count they were
captured for: the one-launch renderer lays its pool of rays out by it. Waves
of 2^30 paths, where the wavefront's queue sizes of one and of five lights are
the same number in 32 bits.

The same paths in both images, so pixels differ by the order of their sums
alone: 1024 samples x (2 + 2 x 5) terms, times 2^-24 below 1e-3."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu


def test_more_lights_in_the_next_frame():
    from illuminaprt_b200.ilg import GpuSpace
    sp = GpuSpace()
    box = scenes.load_box_scene(sp)
    kw = dict(max_depth=2, seed=3, one_launch=True)
    cam = dict(box["camera"], aspect=1.0)
    one = scenes.box_lights(box)
    sp.render(cam, 1024, 1024, 1024, paths_per_wave=1 << 30, **kw)
    sp.set_lights(one * 5)
    got = sp.render(cam, 1024, 1024, 1024, paths_per_wave=1 << 30, **kw)
    want = sp.render(cam, 1024, 1024, 1024, **kw)
    assert want.mean() > 0.01
    assert np.all(np.abs(got - want) <= 1e-3 * np.abs(want) + 1e-6)
    sp.close()
