"""The PLAIN and FP64 forms on the TUNED geometry's pairs (fwd_exact.cu): against the oracle's chain
at the poles, across phi = 0 and on rings wider than the short sine series takes, and the same TOD
bit for bit however the samples' plans are built and ordered.  Tolerances: the forms' own (PLAIN 1e-6
of the TOD rms against the float chain, FP64 1e-12 against the double one)."""
import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _inputs(oracle_mod, nside, nside_beam, radius, n, seed):
    rng = np.random.default_rng(seed)
    sky = rng.normal(size=(4, 12 * nside * nside)).astype(np.float32)
    npix = oracle_mod.beam_npix_for_radius(nside_beam, np.deg2rad(radius))
    from pisco4cmb_gb300 import pix2ang

    theta, phi = pix2ang(nside_beam, np.arange(npix))
    g = np.exp(-0.5 * (theta / np.deg2rad(radius / 2.5)) ** 2)
    maps = np.stack([g, 0.9 * g, 0.1 * g * np.sin(phi), 0.02 * g * np.cos(phi)] * 2).astype(np.float32)
    ra = rng.uniform(0, 2 * np.pi, n)
    dec = np.arcsin(rng.uniform(-1, 1, n))
    r = np.deg2rad(radius)
    k = n // 5
    ra[:k] = rng.uniform(-r, r, k)
    dec[k:2 * k] = np.pi / 2 - rng.uniform(0, 1.5 * r, k)
    dec[2 * k:3 * k] = -np.pi / 2 + rng.uniform(0, 1.5 * r, k)
    dec[:3] = [np.pi / 2, -np.pi / 2, 0.0]
    return sky, npix, maps, ra, dec, rng.uniform(0, np.pi, n)


@pytest.mark.parametrize("nside,nside_beam,radius", [(2, 64, 12.0), (16, 64, 20.0), (64, 256, 5.0),
                                                      (256, 1024, 0.7)])
def test_exact_forms_match_the_chain(gpu, oracle_mod, nside, nside_beam, radius):
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky

    n = 200
    sky, npix, maps, ra, dec, pa = _inputs(oracle_mod, nside, nside_beam, radius, n, nside)
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *sky))
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    conv.update_scan(Scan(n, ra, dec, pa))
    ref = oracle_mod.convolve_f64(ra, dec, pa, nside, sky.astype(np.float64), nside_beam,
                                  maps[:4].astype(np.float64), maps[4:].astype(np.float64))
    for form, tol in (("fp64", 1e-12), ("plain", 1e-6)):
        got = [np.empty(n) for _ in range(2)]
        conv.exec_convolution(*got, form=form)
        for x, y in zip(got, ref):
            assert rel_rms(x, y) < tol, form


@pytest.mark.parametrize("form", ["plain", "fp64"])
def test_exact_forms_do_not_depend_on_the_launch(gpu, oracle_mod, form):
    from pisco4cmb_gb300 import GPUConvolver, RunConfig, Scan, Sky

    nside, n = 64, 9001
    sky, npix, maps, ra, dec, pa = _inputs(oracle_mod, nside, 256, 4.0, n, 5)
    ra[10], dec[11], pa[12] = np.nan, np.inf, np.nan

    def tod(cfg, order="scan", chunk=None):
        conv = GPUConvolver(cfg, form=form)
        conv.update_sky(Sky(nside, *sky.astype(np.float64)))
        conv.set_beam_planes(256, npix, maps[:4].astype(np.float64), maps[4:].astype(np.float64))
        conv.update_scan(Scan(n, ra, dec, pa))
        conv.set_sample_order(order)
        out = [np.empty(n) for _ in range(2)]
        conv.exec_convolution(*out)
        used = conv.memory_used()
        conv.close()
        return out, used

    ref, used = tod(RunConfig())
    assert np.isnan(ref[0][[10, 11, 12]]).all() and np.isfinite(ref[0][:10]).all()
    room = used - 96 * n  # everything but the plans
    for cfg, order in ((RunConfig(ptgPerConv=2000), "scan"), (RunConfig(), "sky"),
                       (RunConfig(maxMemUsage=room + 96 * 2000, ptgPerConv=n), "scan"),
                       (RunConfig(maxMemUsage=room + 96 * 10, ptgPerConv=n), "scan")):
        got, _ = tod(cfg, order)
        for x, y in zip(got, ref):
            assert np.array_equal(x, y, equal_nan=True)
