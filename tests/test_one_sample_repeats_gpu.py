"""One sample a pixel: a pixel has one path, whose contributions are added in
the path's order, so two calls give the same bits: in one launch with any number
of lights, as a wavefront with at most one (it adds to a pixel once a launch and
light), so without a flag, where the size chooses between them, with one. The
sums are those of the wavefront up to their order: at most depth x (lights + 1)
< 150 terms, 150 * 2^-24 = 1e-5, taken as 1e-4 with the few-ulp differences of
the compiler's contractions; a shadow or bounce ray that passes an edge within
such an ulp changes its pixel, one pixel in ten thousand may."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _box(kind):
    from illuminaprt_b200.ilg import GpuSpace
    sp = GpuSpace()
    if kind == "field":
        f = scenes.sphere_field(3, 4, seed=6, width=64, height=64)
        scenes.load_sphere_field(sp, f)
        return sp, f["camera"], f["sky"]
    box = scenes.load_box_scene(sp, scenes.box_scene(specular=kind == "specular", infinite=(0.5, 0.4, 0.3)
                                                     if kind == "infinite" else None))
    if kind in ("two", "eight"):
        sp.set_lights(scenes.box_lights(box) * (2 if kind == "two" else 8))
    elif kind == "dark":
        sp.set_lights([])
    return sp, box["camera"], (0.2, 0.3, 0.4)


@pytest.mark.parametrize("kind", ["box", "specular", "infinite", "two", "eight", "dark", "field"])
def test_images_repeat_bit_for_bit(kind):
    sp, cam, sky = _box(kind)
    for w, h, depth in [(1, 1, 6), (5, 3, 1), (33, 31, 6), (97, 61, 12), (1280, 720, 8)]:
        c = dict(cam, aspect=w / h)
        kw = dict(max_depth=depth, seed=w, sky=sky)
        for one_launch in (False, True) if kind in ("box", "specular", "dark") else (True,):
            first = sp.render(c, w, h, 1, one_launch=one_launch, **kw)
            for _ in range(4):
                assert np.array_equal(sp.render(c, w, h, 1, one_launch=one_launch, **kw), first), (w, h, one_launch)
        assert first.max() > 0
    sp.close()


@pytest.mark.parametrize("kind", ["box", "two", "eight", "dark"])
def test_sums_are_the_wavefronts(kind):
    sp, cam, sky = _box(kind)
    for w, h, depth in [(7, 5, 1), (33, 31, 2), (200, 150, 3)]:
        c = dict(cam, aspect=w / h)
        kw = dict(max_depth=depth, seed=h, sky=sky)
        got, want = sp.render(c, w, h, 1, **kw), sp.render(c, w, h, 1, paths_per_wave=4096, **kw)
        off = np.any(np.abs(got - want) > 1e-4 * np.abs(want) + 1e-6, axis=-1)
        assert off.sum() <= 1 + w * h // 10000, (w, h, depth, off.sum())
    sp.close()


def test_a_batch_with_one_sampled_scenes_repeats():
    from illuminaprt_b200.ilg import GpuSpace
    spaces = [_box(k) for k in ("box", "two", "field")]
    runner = GpuSpace()
    items = [{"space": sp, "camera": dict(cam, aspect=1.0), "width": 48, "height": 48, "spp": spp, "max_depth": 5,
              "seed": 3 + k, "sky": sky} for k, ((sp, cam, sky), spp) in enumerate(zip(spaces, (1, 3, 1)))]
    first = runner.render_batch(items, one_launch=True)
    for _ in range(3):
        again = runner.render_batch(items, one_launch=True)
        for k in (0, 2):  # the scenes with one path a pixel
            assert np.array_equal(again[k], first[k])
        assert np.allclose(again[1], first[1], rtol=1e-4, atol=1e-6)
    for sp, _, _ in spaces:
        sp.close()
    runner.close()
