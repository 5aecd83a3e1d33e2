"""The one-launch renderer against the wavefront at the sizes where its warps'
pools of paths and rays change shape: a single path, fewer paths than a warp,
than a pool (64) and than a block, several pools, paths that end at once
(depth 1), scenes without lights, with the most lights (8) and with an
infinite one. Both trace the same paths; images agree up to the order of the
float additions into a pixel: at most samples x depth x (lights + 1) < 600
terms, 600 * 2^-24 = 4e-5 of the sum, taken as 1e-4 with the few-ulp
differences of the compiler's contractions. A path whose roulette or hit flips
on such an ulp changes its pixel; one pixel in a hundred may."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _space(kind):
    from illuminaprt_b200.ilg import GpuSpace
    sp = GpuSpace()
    if kind == "field":
        f = scenes.sphere_field(2, 3, seed=6, width=64, height=64)
        scenes.load_sphere_field(sp, f)
        return sp, f["camera"], f["sky"]
    box = scenes.load_box_scene(sp, scenes.box_scene(specular=kind == "specular", infinite=(0.5, 0.4, 0.3)
                                                     if kind == "infinite" else None))
    if kind == "dark":
        sp.set_lights([])
    elif kind == "eight":
        sp.set_lights(scenes.box_lights(box) * 8)
    return sp, box["camera"], (0.2, 0.3, 0.4)


@pytest.mark.parametrize("kind", ["box", "specular", "infinite", "dark", "eight", "field"])
def test_one_launch_traces_the_wavefronts_paths(kind):
    sp, cam, sky = _space(kind)
    for w, h, spp, depth in [(1, 1, 1, 6), (5, 3, 2, 1), (13, 5, 1, 9), (31, 33, 3, 2), (97, 61, 2, 6)]:
        kw = dict(max_depth=depth, seed=w, sky=sky)
        c = dict(cam, aspect=w / h)
        wave = sp.render(c, w, h, spp, paths_per_wave=4096, **kw)
        one = sp.render(c, w, h, spp, one_launch=True, **kw)
        again = sp.render(c, w, h, spp, one_launch=True, **kw)
        for img in (one, again):
            off = np.abs(img - wave).max(-1) > 1e-4 * (np.abs(wave).max(-1) + np.abs(wave).mean() + 1e-6)
            assert off.sum() <= max(0, w * h // 100), (kind, w, h, spp, depth, off.sum())
    sp.close()
