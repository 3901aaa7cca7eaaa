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
