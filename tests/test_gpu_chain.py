"""Every form's nearest-lookup TOD against the reference's chain run by its own kernel, which shares
neither the disc nor the pixel decisions with them.  Sky and beam maps are white noise, so that a single
disc or beam pixel that is not the chain's moves its sample's TOD by a few hundredths of the rms.

Tolerances, in units of the TOD's rms, for every sample.  PLAIN: the phasor, good to 1e-12 before it is
rounded to FP32, differs from the chain's in the last bit of one pair in 1e4 (6e-8 of its product): 1e-7.
FP64: the chain's own acos(cos rho) is good to 1e-16 / rho, 1e-10 for a pair at 1e-6 rad, one of some
hundred: 1e-10.  TUNED: FP32's 6e-8 a pair, some 1e-6 / rho at the boresight, 1e-5 at worst."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"plain": 1e-7, "fp64": 1e-10, "tuned": 1e-5}


def _setup(nside, nside_beam, radius, n, seed, double=False):
    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky, beam_npix_for_radius

    rng = np.random.default_rng(seed)
    kind = np.float64 if double else np.float32
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *rng.normal(size=(4, 12 * nside * nside)).astype(kind)))
    npix = beam_npix_for_radius(nside_beam, np.deg2rad(radius))
    maps = rng.normal(size=(8, npix)).astype(kind)
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    r = np.deg2rad(radius)
    ra = rng.uniform(-20.0, 20.0, n)
    dec = np.arcsin(rng.uniform(-1, 1, n))
    k = n // 8
    ra[:k] = rng.uniform(-r, r, k)
    dec[k:2 * k] = np.pi / 2 - rng.uniform(0, 1.5 * r, k)
    dec[2 * k:3 * k] = -np.pi / 2 + rng.uniform(0, 1.5 * r, k)
    dec[3 * k:4 * k] = np.deg2rad(rng.uniform(76, 89, k))
    dec[:4] = [np.pi / 2, -np.pi / 2, 0.0, np.pi / 2 - r]
    conv.update_scan(Scan(n, ra, dec, rng.uniform(-np.pi, np.pi, n)))
    return conv


def _tod(call, n, f64=True):
    import torch

    out = torch.full((2, n), float("nan"), dtype=torch.float64 if f64 else torch.float32, device="cuda")
    torch.cuda.synchronize()
    call(out)
    return out


@pytest.mark.parametrize("nside,nside_beam,radius,n,double", [
    (1, 64, 25.0, 4000, False), (3, 50, 20.0, 4001, True), (16, 64, 20.0, 4000, False),
    (64, 256, 5.0, 8000, True), (100, 300, 3.0, 3001, False), (256, 1024, 4.0, 2000, False),
    (512, 512, 1.0, 3000, False), (1024, 2048, 3.0, 300, False), (2048, 8192, 1.0, 300, True)])
def test_forms_follow_the_chain(gpu, nside, nside_beam, radius, n, double):
    conv = _setup(nside, nside_beam, radius, n, nside, double)
    for form, tol in TOL.items():
        chain = "plain" if form == "plain" else "fp64"
        if form == "tuned" and double:  # its maps are the FP32 ones
            continue
        ref = _tod(lambda t: (conv.debug_forward_chain(t[0].data_ptr(), t[1].data_ptr(), form=chain),
                              conv.sync()), n)
        rms = ref.std().item()
        for order in ("scan", "sky"):
            conv.set_sample_order(order)
            got = _tod(lambda t: (conv.forward_device(t[0].data_ptr(), t[1].data_ptr(), out_f64=True,
                                                      form=form), conv.sync()), n)
            assert (got - ref).abs().max().item() < tol * rms, (form, order)
        conv.set_sample_order("scan")
    conv.close()


def test_chain_is_the_bilinear_forms_own_kernel(gpu):
    """With the bilinear lookup PLAIN and FP64 run the chain: the same bits; TUNED is refused."""
    import torch

    from pisco4cmb_gb300 import PiscoInvalidArgument

    n = 1500
    conv = _setup(64, 256, 4.0, n, 2)
    conv.set_interp(True)
    for form in ("plain", "fp64"):
        ref = _tod(lambda t: (conv.debug_forward_chain(t[0].data_ptr(), t[1].data_ptr(), form=form),
                              conv.sync()), n)
        got = _tod(lambda t: (conv.forward_device(t[0].data_ptr(), t[1].data_ptr(), out_f64=True,
                                                  form=form), conv.sync()), n)
        assert torch.equal(got, ref)
    with pytest.raises(PiscoInvalidArgument):
        conv.debug_forward_chain(0, 0, form="tuned")
    conv.close()


def test_longest_rings_follow_the_chain(gpu):
    """nside 8192, rings of 2^15 pixels: PLAIN and TUNED against PLAIN's chain (TUNED: both round to
    FP32), and every pair's pixel."""
    import torch

    from pisco4cmb_gb300 import GPUConvolver, Scan, beam_npix_for_radius

    nside, n = 8192, 300
    g = torch.Generator("cuda").manual_seed(1)
    sky = torch.randn((12 * nside * nside, 4), generator=g, device="cuda")
    conv = GPUConvolver()
    conv.set_sky_device(nside, sky.data_ptr(), False, stream=1)
    torch.cuda.synchronize()
    del sky
    torch.cuda.empty_cache()
    rng = np.random.default_rng(2)
    npix = beam_npix_for_radius(8192, np.deg2rad(0.25))
    maps = rng.normal(size=(8, npix)).astype(np.float32)
    conv.set_beam_planes(8192, npix, maps[:4], maps[4:])
    dec = np.concatenate([rng.uniform(-0.7, 0.7, n - 80), np.pi / 2 - rng.uniform(0, 5e-3, 40),
                          rng.uniform(1.3, 1.55, 40)])
    conv.update_scan(Scan(n, rng.uniform(-5e-3, 5e-3, n), dec, rng.uniform(0, np.pi, n)))
    ref = _tod(lambda t: (conv.debug_forward_chain(t[0].data_ptr(), t[1].data_ptr(), form="plain"),
                          conv.sync()), n)
    for form in ("plain", "tuned"):
        got = _tod(lambda t: (conv.forward_device(t[0].data_ptr(), t[1].data_ptr(), out_f64=True, form=form),
                              conv.sync()), n)
        assert (got - ref).abs().max().item() < TOL[form] * ref.std().item(), form
        check = conv.debug_decisions(form)
        assert check.pairs == conv.count_pairs() and check.differing == 0
        assert check.worst_fp32 < 0.5 and check.worst_fp64 < 0.5
    conv.close()
