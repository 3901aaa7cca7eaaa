"""Rounding errors of the kernels against their floor, with tolerances from the number of roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_tuned_sum_rounds_once_per_pair(gpu):
    """A sky of I with faint Q, U and V: a pair's product is rounded once at I's magnitude.

    One rounding of a value with an evenly spread logarithm has a relative rms of 2^-24 sqrt(0.541 / 3)
    = 2.53e-8; a sample's total of n pairs t is off by 2.53e-8 sqrt(n <t^2>) rms (its own sum is
    compensated, the output float64).  The parts at the faint components' magnitude are 1e-3 of it.  Two
    roundings give 1.41 times that, three 1.73; the line is 1.2."""
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky, beam_npix_for_radius

    nside, nside_beam, n = 64, 256, 20_000
    rng = np.random.default_rng(4)
    npix = 12 * nside * nside
    stokes = [rng.uniform(50.0, 150.0, npix)] + [rng.uniform(-0.1, 0.1, npix) for _ in range(3)]
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *[s.astype(np.float32) for s in stokes]))
    nb = beam_npix_for_radius(nside_beam, np.deg2rad(5.0))
    maps = rng.uniform(0.5, 1.5, (8, nb)).astype(np.float32)
    conv.set_beam_planes(nside_beam, nb, maps[:4], maps[4:])
    conv.update_scan(Scan(n, rng.uniform(0, 2 * np.pi, n), np.arcsin(rng.uniform(-0.9, 0.9, n)),
                          rng.uniform(0, np.pi, n)))
    ref, got = [[np.empty(n) for _ in range(2)] for _ in range(2)]
    conv.exec_convolution(*ref, form="fp64")
    conv.exec_convolution(*got, form="tuned")
    pairs = conv.count_pairs() / n
    mean_square = (100.0 ** 2 + 100.0 ** 2 / 12.0) * (1.0 + 1.0 / 12.0)
    floor = 2.53e-8 * np.sqrt(pairs * mean_square)
    for x, y in zip(got, ref):
        assert np.sqrt(np.mean((x - y) ** 2)) < 1.2 * floor


@pytest.mark.parametrize("widest", [np.pi, 60.0])
def test_map_sines_are_rounded_once(gpu, widest):
    """cos and sin of 2 psi in the normal equations (one value per pixel): a result that is the rounded
    sum of a table entry and a small correction is off by 0.29 ulp rms; near a zero (some 5 % of the
    angles) the correction is as large as the result and its own rounding comes on top: at most 1 ulp and
    the series' 1e-2."""
    import torch

    from pisco4cmb_gb300 import SkyMap, pix2ang

    nside = 64
    npix = 12 * nside * nside
    theta, phi = pix2ang(nside, np.arange(npix))
    pa = np.random.default_rng(6).uniform(-widest, widest, npix)
    m = SkyMap(nside)
    dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (phi, np.pi / 2 - theta, pa, np.ones(npix))]
    m.accumulate_device(npix, *[v.data_ptr() for v in dev[:3]], 1, np.zeros(1, np.float32), dev[3].data_ptr(),
                        f64=True, stream=1)
    ata = m.get_normal()[0].reshape(npix, 9)
    wide = np.longdouble(2.0 * -pa)
    assert np.finfo(np.longdouble).eps < 2e-19
    for got, ref in ((ata[:, 1], np.cos(wide)), (ata[:, 2], np.sin(wide))):
        ulp = np.spacing(np.abs(ref).astype(np.float64))
        err = np.abs((np.longdouble(got) - ref) / ulp).astype(np.float64)
        assert np.sqrt(np.mean(err ** 2)) < 0.34
        assert err.max() < 1.1
