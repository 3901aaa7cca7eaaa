"""The longitude's reduction to four quarter turns in two floats, as the map-maker's FP32 pixel makes it
(skymap.cu quick_ang2pix): th + turns rounds for th in (-2, 0), and the two parts together must not."""
import numpy as np
import pytest

F, D = np.float32, np.float64


def _reduce(ra):
    """tt, tl of longitudes: quarter turns mod 4."""
    rh = ra.astype(F)
    rl = (ra - rh.astype(D)).astype(F)
    k = F(0.63661975)
    th = rh * k
    turns = F(-4.0) * np.floor(F(0.25) * th)
    tt = th + turns
    fma = lambda a, b, c: (D(a) * D(b) + D(c)).astype(F)  # noqa: E731 -- the product is exact in FP64
    tl = fma(rl, k, fma(rh, F(2.56825533e-8), fma(rh, k, -th))) + (th - (tt - turns))
    return tt, tl


@pytest.mark.parametrize("lo,hi", [(0.0, 2.0 * np.pi), (-np.pi, 0.0), (-1e-3, 1e-3), (-1e4, 1e4)])
def test_two_floats_hold_the_longitude(lo, hi):
    ra = np.random.default_rng(3).uniform(lo, hi, 1_000_000)
    tt, tl = _reduce(ra)
    assert tt.dtype == tl.dtype == F
    turns = D(ra) * (2.0 / np.pi)
    err = tt.astype(D) + tl.astype(D) - turns
    err -= 4.0 * np.round(err / 4.0)
    # 2/pi as two floats leaves 1e-15 of ra; tl, at most 3e-4, is rounded to 2^-24 a few times; the
    # FP64 product here to 2^-53 of 6400
    assert np.abs(err).max() < 1e-10 + 3 * 2.0 ** -24 * np.abs(tl).max() + 1e-12


def test_without_the_remainder_a_negative_longitude_loses_digits():
    ra = np.random.default_rng(3).uniform(-np.pi, 0.0, 1_000_000)
    th = ra.astype(F) * F(0.63661975)
    tt = th + F(4.0)
    lost = np.abs(th - (tt - F(4.0)))
    assert lost.max() > 1.1e-7  # two thirds of what the pixel's error bound allows in all
