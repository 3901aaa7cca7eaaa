"""The map-maker's pixel of a pointing (FP32 with the FP64 decision near an edge, skymap.cu): the hit
map equals the counts of the oracle's ang2pix, for pointings all over the sky, at both poles, at the
caps' border and on pixel edges (each edge pointing nudged by up to 1e-9 rad)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside", [1, 2, 16, 512, 4096])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_hits_equal_the_oracle(gpu, oracle_mod, nside, dtype):
    import torch

    from pisco4cmb_gb300 import SkyMap

    rng = np.random.default_rng(nside)
    n = 60000
    ra = rng.uniform(-2 * np.pi, 4 * np.pi, n)
    dec = np.arcsin(rng.uniform(-1, 1, n))
    k = n // 6
    dec[:k] = np.pi / 2 - rng.uniform(0, 3.0 / nside, k).clip(0, 1)
    dec[k:2 * k] = -np.pi / 2 + rng.uniform(0, 3.0 / nside, k).clip(0, 1)
    dec[2 * k:3 * k] = np.arcsin(2.0 / 3.0) + rng.uniform(-2e-6, 2e-6, k)
    # equatorial edges: nside (1/2 + 2 ra / pi) - 3/4 nside z an integer
    z = rng.uniform(-0.66, 0.66, k)
    j = rng.integers(0, 4 * nside, k)
    ra[3 * k:4 * k] = ((j + 0.75 * nside * z) / nside - 0.5) * (np.pi / 2) + rng.uniform(-1e-9, 1e-9, k)
    dec[3 * k:4 * k] = np.arcsin(z)
    dec[:4] = [np.pi / 2, -np.pi / 2, 0.0, np.pi / 4]
    ra[:4] = [0.0, 1.0, np.pi / 2, -np.pi]
    ra, dec = ra.astype(dtype), dec.astype(dtype)
    half = dtype(np.pi / 2)
    if float(half) > np.pi / 2:
        half = np.nextafter(half, dtype(0))
    dec = dec.clip(-half, half)
    pa = rng.uniform(0, np.pi, n).astype(dtype)
    want = oracle_mod.ang2pix(nside, np.pi / 2 - dec.astype(np.float64), ra.astype(np.float64))
    m = SkyMap(nside)
    t = [torch.from_numpy(v).cuda() for v in (ra, dec, pa, np.ones(n, dtype))]
    m.accumulate_device(n, *[v.data_ptr() for v in t[:3]], 1, [0.0], t[3].data_ptr(),
                        f64=dtype is np.float64, stream=1)
    npix = m.size()

    class View:
        __cuda_array_interface__ = dict(shape=(npix,), typestr="<f8", data=(m.device_arrays()[2], False),
                                        version=3)

    hits = torch.as_tensor(View(), device="cuda").cpu().numpy()
    pix, count = np.unique(want, return_counts=True)
    assert np.array_equal(np.flatnonzero(hits), pix)
    assert np.array_equal(hits[pix], count)
    m.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("longest", [1, 7, 200])
def test_totals_do_not_depend_on_how_pixels_are_reduced(gpu, dtype, longest):
    """A pixel's totals are its values added one by one in order, whether one thread adds them (few
    values per occupied pixel) or eight lanes do (many): the same bits with and without other pixels
    of one value each in the call."""
    from pisco4cmb_gb300 import SkyMap, pix2ang

    nside = 64
    rng = np.random.default_rng(longest)
    few = rng.permutation(np.repeat(np.arange(100, 140), rng.integers(longest, longest + 5, 40)))
    many = np.arange(4000, 4000 + 2 * len(few) + 300)

    def normal(pix, pa, data):
        theta, phi = pix2ang(nside, pix)
        m = SkyMap(nside)
        n = len(pix)
        m.accumulate_data(n, *[v.astype(dtype)[None] for v in (phi, np.pi / 2 - theta, pa)], 1,
                          np.array([0.3], np.float32), data.astype(dtype)[None])
        got = [v.reshape(12 * nside * nside, -1)[100:140] for v in m.get_normal()]
        m.close()
        return got

    pa, data = rng.uniform(0, np.pi, len(few)), rng.normal(size=len(few))
    pa2, data2 = rng.uniform(0, np.pi, len(many)), rng.normal(size=len(many))
    alone = normal(few, pa, data)
    mixed = normal(np.concatenate([few, many]), np.concatenate([pa, pa2]),
                   np.concatenate([data, data2]))
    for x, y in zip(alone, mixed):
        assert x.any(axis=1).all() and np.array_equal(x, y)
