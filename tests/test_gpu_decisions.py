"""The decisions of the forms' own pair loops against the reference's FP64 chain, pair by pair on the
device: the beam pixel of every disc pair is the chain's, and no FP32 decision is off by more than half
of the margin within which it is redone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# sky nside, beam nside, beam radius, declinations: longitude offsets from a few degrees to the whole circle
SHAPES = [(64, 256, 5.0, (-60.0, 60.0), 60_000), (64, 256, 5.0, (76.0, 89.0), 60_000),
          (256, 1024, 4.0, (60.0, 89.9), 6_000), (16, 64, 20.0, (-90.0, 90.0), 30_000),
          (1024, 2048, 3.0, (-85.0, 85.0), 400), (2048, 4096, 1.0, (80.0, 90.0), 1_000)]


def convolver(nside, nside_beam, radius, decs, n, seed=11):
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky, beam_npix_for_radius

    rng = np.random.default_rng(seed)
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *rng.normal(size=(4, 12 * nside * nside)).astype(np.float32)))
    npix = beam_npix_for_radius(nside_beam, np.deg2rad(radius))
    maps = rng.normal(size=(8, npix)).astype(np.float32)
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    conv.update_scan(Scan(n, rng.uniform(0, 2 * np.pi, n), np.deg2rad(rng.uniform(*decs, n)),
                          rng.uniform(0, np.pi, n)))
    return conv


@pytest.mark.parametrize("form", ["tuned", "fp64", "plain"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_decisions_are_the_chains(gpu, shape, form):
    conv = convolver(*shape)
    got = conv.debug_decisions(form)
    assert got.pairs == conv.count_pairs()
    assert got.differing == 0
    assert got.worst_fp32 < 0.5
    conv.close()


def test_reevaluation_is_the_chains(gpu):
    """Pairs from 1e-4 to 3e-3 rad from the boresight on the finest beam grid, where acos(cos rho)
    makes the chain's own rounding largest: what the FP64 re-evaluation decides by itself differs from
    the chain by less than half of the margin within which it leaves the decision to the chain."""
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky, beam_npix_for_radius, pix2ang

    nside, nside_beam, n = 64, 8192, 300_000
    rng = np.random.default_rng(12)
    theta, phi = pix2ang(nside, rng.integers(2 * nside * (nside - 1), 10 * nside * nside, n))
    rho = np.exp(rng.uniform(np.log(1e-4), np.log(3e-3), n))
    turn = rng.uniform(0, 2 * np.pi, n)
    dec = np.pi / 2 - theta + rho * np.cos(turn)
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *rng.normal(size=(4, 12 * nside * nside)).astype(np.float32)))
    npix = beam_npix_for_radius(nside_beam, np.deg2rad(0.5))
    maps = rng.normal(size=(8, npix)).astype(np.float32)
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    conv.update_scan(Scan(n, phi + rho * np.sin(turn) / np.cos(dec), dec, rng.uniform(0, np.pi, n)))
    got = conv.debug_decisions("tuned")
    assert got.pairs >= n
    assert got.differing == 0
    assert got.worst_fp64 < 0.5
    conv.close()
