"""A short TUNED launch's blocks, in both shapes and on either side of every line between them: the TOD
of a range equals that of the same samples in a long launch, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bilinear", [False, True])
def test_short_launches_are_one_result(gpu, bilinear):
    import torch

    from pisco4cmb_gb300 import GPUConvolver, Scan, Sky, beam_npix_for_radius

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(8)
    nside, nside_beam, total = 64, 256, 80 * sms
    conv = GPUConvolver()
    conv.update_sky(Sky(nside, *rng.normal(size=(4, 12 * nside * nside)).astype(np.float32)))
    npix = beam_npix_for_radius(nside_beam, np.deg2rad(4.0))
    maps = rng.normal(size=(8, npix)).astype(np.float32)
    conv.set_beam_planes(nside_beam, npix, maps[:4], maps[4:])
    conv.update_scan(Scan(total, rng.uniform(0, 2 * np.pi, total), np.arcsin(rng.uniform(-1, 1, total)),
                          rng.uniform(0, np.pi, total)))
    conv.set_interp(bilinear)

    def tod(begin, n):
        out = torch.full((2, n), float("nan"), device="cuda")
        torch.cuda.synchronize()
        conv.forward_device(out[0].data_ptr(), out[1].data_ptr(), begin=begin, n=n)
        conv.sync()
        return out

    whole = tod(0, total)
    assert not whole.isnan().any()
    # samples per block (two blocks per SM), its neighbours by one, and launches smaller than a block each
    for share in (1, 8, 10, 16, 20, 24, 30, 32):
        for n in (2 * sms * share - 1, 2 * sms * share, 2 * sms * share + 1):
            got = tod(7, n)
            assert torch.equal(got, whole[:, 7:7 + n]), n
    for n in (1, 2, 31, 33, sms):
        assert torch.equal(tod(3, n), whole[:, 3:3 + n])
    conv.close()
