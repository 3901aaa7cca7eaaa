"""The TUNED forward with two pixels per lane, where its packing could go wrong: discs whose ranges
start and end on either parity, wrap at phi = 0, hold one pixel or whole rings (both poles, tiny
skies), rings of up to 2^15 pixels (their ends share one word), and a sky that is only 16-byte
aligned.  Reference: the FP64 form; tolerance: the TUNED form's own, 1e-6 of the TOD rms."""
import ctypes

import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _beam(rng, nside_beam, radius_deg):
    from pisco4cmb_gb300 import beam_npix_for_radius, pix2ang

    npix = beam_npix_for_radius(nside_beam, np.deg2rad(radius_deg))
    theta, phi = pix2ang(nside_beam, np.arange(npix))
    g = np.exp(-0.5 * (theta / np.deg2rad(radius_deg / 2.5)) ** 2)
    return npix, np.stack([g, 0.9 * g, 0.1 * g * np.sin(phi), 0.02 * g * np.cos(phi)] * 2).astype(np.float32)


def _run(conv, n, form):
    out = [np.empty(n, np.float64) for _ in range(2)]
    conv.exec_convolution(*out, form=form)
    return out


@pytest.mark.parametrize("nside,nside_beam,radius", [(1, 64, 25.0), (2, 64, 12.0), (4, 128, 2.0),
                                                      (16, 64, 20.0), (64, 128, 5.0), (512, 512, 1.0)])
def test_two_pixels_per_lane_edges(gpu, nside, nside_beam, radius):
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky

    rng = np.random.default_rng(nside)
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *rng.normal(size=(4, 12 * nside * nside)).astype(np.float32)))
    npix, maps = _beam(rng, nside_beam, radius)
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    n = 1500
    ra = rng.uniform(-np.pi, 3 * np.pi, n)
    dec = np.arcsin(rng.uniform(-1, 1, n))
    r = np.deg2rad(radius)
    ra[:400] = rng.uniform(-r, r, 400)                       # wrap at phi = 0
    dec[400:500] = np.pi / 2 - rng.uniform(0, r, 100)        # the north pole inside the disc
    dec[500:600] = -np.pi / 2 + rng.uniform(0, r, 100)       # the south pole
    dec[600:604] = [np.pi / 2, -np.pi / 2, 0.0, np.pi / 2 - r]
    conv.update_scan(Scan(n, ra, dec, rng.uniform(0, np.pi, n)))
    ref = _run(conv, n, "fp64")
    got = _run(conv, n, "tuned")
    for x, y in zip(got, ref):
        assert rel_rms(x, y) < 1e-6


def test_longest_rings(gpu):
    """nside 8192: rings of 2^15 pixels, ranges that end beyond 2^15."""
    import torch

    from pisco4cmb_gb300 import GPUConvolver, Scan

    nside = 8192
    g = torch.Generator("cuda").manual_seed(1)
    sky = torch.randn((12 * nside * nside, 4), generator=g, device="cuda")
    conv = GPUConvolver()
    conv.set_sky_device(nside, sky.data_ptr(), False, stream=1)
    torch.cuda.synchronize()
    del sky
    rng = np.random.default_rng(2)
    npix, maps = _beam(rng, 8192, 0.25)
    conv.set_beam_planes(8192, npix, maps[:4], maps[4:])
    n = 300
    ra = rng.uniform(-5e-3, 5e-3, n)
    dec = np.concatenate([rng.uniform(-0.7, 0.7, n - 40), np.pi / 2 - rng.uniform(0, 5e-3, 40)])
    conv.update_scan(Scan(n, ra, dec, rng.uniform(0, np.pi, n)))
    got = _run(conv, n, "tuned")
    ref = _run(conv, n, "plain")
    for x, y in zip(got, ref):
        assert rel_rms(x, y) < 1e-6
    conv.close()


@pytest.mark.parametrize("offset", [0, 4])
def test_sky_alignment(gpu, offset):
    """pisco_forward_batched_noalloc takes a sky at any 16-byte boundary: 32 bytes are not assumed."""
    import torch

    from pisco4cmb_gb300 import _lib

    nside, nside_beam, n = 32, 128, 700
    rng = np.random.default_rng(3)
    npix, maps = _beam(rng, nside_beam, 4.0)
    flat = torch.zeros(48 * nside * nside + 8, device="cuda")
    assert flat.data_ptr() % 32 == 0
    sky = flat[offset:offset + 48 * nside * nside]
    sky.copy_(torch.from_numpy(rng.normal(size=48 * nside * nside).astype(np.float32)))
    beam = torch.from_numpy(np.ascontiguousarray(maps.T)).cuda()
    scan = [torch.from_numpy(v).cuda() for v in (rng.uniform(0, 2 * np.pi, n),
                                                  np.arcsin(rng.uniform(-1, 1, n)),
                                                  rng.uniform(0, np.pi, n))]
    tod = torch.empty((2, n), device="cuda")
    det = (_lib.NoallocDet * 1)(_lib.NoallocDet(nside_beam, npix, beam.data_ptr(), n,
                                                *[v.data_ptr() for v in scan], tod[0].data_ptr(),
                                                tod[1].data_ptr()))
    torch.cuda.synchronize()
    lib = _lib.load()
    _lib.check(lib.pisco_forward_batched_noalloc(0, nside, ctypes.c_void_p(sky.data_ptr()), det, 1, 0, 1),
               None, "noalloc")
    from pisco4cmb_gb300 import GPUConvolver

    conv = GPUConvolver()
    conv.set_sky_device(nside, sky.data_ptr(), False, stream=1)
    conv.set_beam_device(nside_beam, npix, beam.data_ptr(), stream=1)
    conv.set_scan_device(n, *[v.data_ptr() for v in scan], stream=1)
    ref = torch.empty((2, n), device="cuda")
    conv.forward_device(ref[0].data_ptr(), ref[1].data_ptr(), stream=1)
    conv.sync()
    assert torch.equal(tod, ref)
