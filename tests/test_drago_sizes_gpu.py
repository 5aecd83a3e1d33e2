"""DragoTone on the device against its formula in numpy (logarithms and powers
in double, rounded to float, as the device does), from one pixel to several
blocks of the maximum's reduction.

The two differ where a double logarithm's last bit moves a float rounding: at
most one float step in each of the factors, four steps of the quotient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _log10(x):
    return np.log10(x.astype(np.float64)).astype(F)


def _drago(img):
    top = img.reshape(-1, 3).max(axis=0)
    scale = F(95) * F(0.01)
    bias = F(np.log10(np.float64(F(0.8)))) / F(np.log10(np.float64(F(0.5))))
    a = scale / (np.log((top + F(1)).astype(np.float64)) / np.log(10.0)).astype(F)
    power = np.power((img / top).astype(np.float64), np.float64(bias)).astype(F)
    out = a * _log10(img + F(1)) / _log10(F(2) + power * F(8))
    return np.clip(out, F(0), F(1))


@pytest.mark.parametrize("shape", [(1, 1), (1, 3), (15, 17), (16, 16), (257, 3), (301, 999)])
def test_drago_matches_its_formula(shape):
    from illuminaprt_b200.ilg import GpuSpace
    img = (np.random.default_rng(shape[1]).random((*shape, 3)) ** 3 * 20.0 + 1e-3).astype(F)
    sp = GpuSpace()
    got = sp.tonemap(img, "drago")
    sp.close()
    assert np.abs(got - _drago(img)).max() <= 4 * 2.0 ** -23
