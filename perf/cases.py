"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" says which entry point it goes through:

  forward   GPUConvolver.forward_device: resident pointing in, TOD a and b out (any form, beam lookup
            and sample order)
  host      GPUConvolver.update_scan + exec_convolution: host pointing in, host TOD out
  batched   GPUConvolver.forward_batched: a focal plane of uneven detector pairs
  maps      autograd.convolve, forward and backward: TOD, sky gradient and beam-map gradient
  params    autograd.convolve_gaussian, forward and backward: TOD, sky gradient and the gradient of the
            beam's five parameters
  adjoint   GPUConvolver.adjoint_device: TOD residuals back onto the sky
  mapmake   SkyMap: TOD accumulated into normal equations, solved for I, Q, U
  pointing  pisco_focal_plane_to_sky_device: every detector's pointing from the array centre's

Sizes are those of the repository's five workloads (nside 64 to 2048 skies, beams of 1 to 5 degrees)
with as many samples as keep a pass between a fraction of a millisecond and some tens of them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pisco4cmb_gb300 import GPUConvolver, PolBeam, Scan, SkyMap
from pisco4cmb_gb300 import _lib
from pisco4cmb_gb300.autograd import convolve, convolve_gaussian

F64 = torch.float64
PI = math.pi
EPSILON = 0.01
MOST_PAIRS = 3.5e9  # of a TUNED pass with the nearest lookup: the largest listed case
# cost of a pair of the other paths, in such pairs
COST = {"tuned": 1.0, "bilinear": 2.4, "plain": 110.0, "fp64": 120.0, "maps": 6.0, "params": 3.0, "adjoint": 2.0}
FLOPS = 110.0  # of a pair: its place in the beam's frame, beam pixel, rotation and two sums


def listed():
    return [
        # the next half sweep of an observation as it streams in: a short launch, where latency counts
        dict(name="stream", kind="forward", form="tuned", bilinear=False, order="scan", scan="sweep",
             nside=1024, nside_beam=2048, radius=3.0, n=2003),
        # a survey at production size: nside 1024 sky, 3 degree beam, constant-elevation sweeps
        dict(name="survey", kind="forward", form="tuned", bilinear=False, order="scan", scan="sweep",
             nside=1024, nside_beam=2048, radius=3.0, n=400_000),
        # a high-resolution sky (larger than L2) with a narrow beam and a tenth of the pointings at the
        # poles, taken in sky order
        dict(name="high_resolution", kind="forward", form="tuned", bilinear=False, order="sky",
             scan="poles", nside=2048, nside_beam=4096, radius=1.0, n=300_001),
        # the survey with the interpolated beam
        dict(name="interpolated", kind="forward", form="tuned", bilinear=True, order="scan",
             scan="sweep", nside=1024, nside_beam=2048, radius=3.0, n=100_003),
        # a run of the reference's own size on its per-pair chain, from host arrays to host arrays in
        # float64: what a caller of its Convolver has
        dict(name="drop_in", kind="host", form="plain", scan="raster", nside=64, nside_beam=256,
             radius=5.0, n=20_000),
        # the all-FP64 form on a part of a scan: the check of a production run's precision
        dict(name="all_fp64", kind="forward", form="fp64", bilinear=False, order="scan", scan="poles",
             nside=2048, nside_beam=4096, radius=1.0, n=6_001),
        # a focal plane: 48 detector pairs, beams of 1 to 5 degrees, uneven sample counts, one launch
        dict(name="focal_plane", kind="batched", nside=512, nside_beam=1024, ndet=48, least=2_000,
             most=100_000),
        # a step of a sky and beam-map fit: forward and bit-reproducible backward
        dict(name="fit_maps", kind="maps", nside=256, nside_beam=1024, radius=4.0, n=200_000),
        # a step of a sky and beam-parameter fit
        dict(name="fit_parameters", kind="params", nside=256, nside_beam=1024, radius=4.0, n=200_000),
        # the back-projection of an iterative map-maker, with float atomics
        dict(name="back_project", kind="adjoint", deterministic=False, nside=1024, nside_beam=2048,
             radius=3.0, n=40_009),
        # four detectors' TOD binned into maps
        dict(name="bin_maps", kind="mapmake", nside=512, ndet=4, n=250_007),
        # a focal plane's pointing from the array centre's
        dict(name="detector_pointing", kind="pointing", ndet=96, n=30_011),
    ]


def draw(rng):
    kind = rng.choice(["forward"] * 5 + ["host", "batched", "maps", "params", "adjoint", "mapmake",
                                         "pointing"])

    def spread(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    if kind == "mapmake":
        return dict(kind=kind, nside=rng.choice([64, 128, 256, 512, 1024]), ndet=rng.randint(3, 8),
                    n=int(spread(2e3, 1.5e5)))
    if kind == "pointing":
        return dict(kind=kind, ndet=rng.randint(1, 96), n=int(spread(1e3, 3e4)))
    if kind == "batched":
        return dict(kind=kind, nside=rng.choice([128, 256, 512]), nside_beam=1024,
                    ndet=rng.randint(2, 48), least=1_000, most=int(spread(2e3, 1e5)))
    case = dict(kind=kind)
    nside = rng.choice([64, 256, 512, 1024, 2048] if kind == "forward" else
                       [64, 128] if kind == "host" else [64, 256, 512, 1024])
    radius = round(spread(1.0, 5.0), 3)
    cost = 1.0
    if kind == "forward":
        form = rng.choice(["tuned", "tuned", "tuned", "plain", "fp64"])
        bilinear = rng.random() < 0.35
        cost = COST[form] * (COST["bilinear"] if bilinear else 1.0)
        case |= dict(form=form, bilinear=bilinear, order=rng.choice(["scan", "scan", "sky"]),
                     scan=rng.choice(["sweep", "sweep", "poles", "raster"]))
    elif kind == "host":
        case |= dict(form=rng.choice(["plain", "tuned"]), scan="raster")
        cost = COST[case["form"]]
    else:
        cost = COST[kind]
        if kind == "adjoint":
            case |= dict(deterministic=rng.random() < 0.5)
    case |= dict(nside=nside, nside_beam=rng.choice([2, 4]) * max(nside, 128), radius=radius)
    per = max(1.0, 6.0 * nside * nside * (1.0 - math.cos(math.radians(radius))))
    most = min(400_000.0, MOST_PAIRS / cost / per)
    return case | dict(n=int(spread(min(500.0, most / 4), most)))


# ---------------------------------------------------------------- inputs
def _generator(seed, what):
    return torch.Generator("cuda").manual_seed((int(seed) * 1009 + what) % (1 << 62))


def _rings(nside):
    """z, pixels, half-pixel shift and first pixel of every RING-scheme ring (ring 1 at index 0)."""
    i = torch.arange(1, 4 * nside, dtype=torch.int64, device="cuda")
    north = torch.where(i > 2 * nside, 4 * nside - i, i)
    cap = north < nside
    fn = north.to(F64)
    z = torch.where(cap, 1.0 - fn * fn / (3.0 * nside * nside), (2.0 * nside - fn) * 2.0 / (3.0 * nside))
    z = torch.where(i > 2 * nside, -z, z)
    count = torch.where(cap, 4 * north, torch.full_like(north, 4 * nside))
    shift = torch.where(cap, 0.5, torch.where((north - nside) % 2 == 0, 0.5, 0.0)).to(F64)
    start = torch.cumsum(count, 0) - count
    return z, count, shift, start


def _sky(nside, seed):
    """npix x 4 float32 I, Q, U, V in microkelvin: plane waves with amplitude ~ 1 / k and white noise,
    I of 100 and Q, U of 10 rms, V = 0."""
    z, count, shift, start = _rings(nside)
    g = _generator(seed, 1)
    npix = 12 * nside * nside
    sky = torch.zeros((npix, 4), device="cuda")
    row = torch.repeat_interleave(torch.arange(z.numel(), device="cuda"), count)
    j = torch.arange(npix, device="cuda") - start[row]
    phi = ((j.to(F64) + shift[row]) * (2.0 * PI / count.to(F64)[row])).float()
    zf = z.float()[row]
    s = torch.sqrt((1.0 - zf) * (1.0 + zf))
    x, y = s * torch.cos(phi), s * torch.sin(phi)
    del row, j, phi, s
    waves = 8
    for c, rms in enumerate((100.0, 10.0, 10.0)):
        k = 2.0 * (min(200.0, nside) / 2.0) ** torch.rand(waves, generator=g, device="cuda")
        d = torch.nn.functional.normalize(torch.randn(waves, 3, generator=g, device="cuda"), dim=1)
        p = 2.0 * PI * torch.rand(waves, generator=g, device="cuda")
        m = torch.zeros(npix, device="cuda")
        for w in range(waves):
            kw = k[w] * d[w]
            m += torch.cos(kw[0] * x + kw[1] * y + kw[2] * zf + p[w]) / k[w]
        m *= 1.0 / m.std()
        m += 0.1 * torch.randn(npix, generator=g, device="cuda")
        sky[:, c] = rms * m
    return sky


def _beam_pixels(nside_beam, radius_deg):
    """Pixels of a beam map of that radius, and their theta and phi (float64)."""
    top = int(nside_beam * math.sqrt(3.0 * (1.0 - math.cos(math.radians(radius_deg)))))
    ring = torch.arange(1, top + 1, device="cuda")
    i = torch.repeat_interleave(ring, 4 * ring)
    npix = 2 * top * (top + 1)
    j = torch.arange(npix, device="cuda") - 2 * i * (i - 1)
    t = i.to(F64) ** 2 / (3.0 * nside_beam * nside_beam)
    theta = torch.atan2(torch.sqrt(t * (2.0 - t)), 1.0 - t)
    return npix, theta, (j.to(F64) + 0.5) * (0.5 * PI) / i.to(F64)


def _beam(nside, nside_beam, radius_deg, fwhm_deg, ellipticity, seed):
    """npix x 8 float32 (a.IQUV, b.IQUV): elliptical Gaussians with 1 % cross-polar leakage, normalised
    as PolBeam.build does."""
    npix, theta, phi = _beam_pixels(nside_beam, radius_deg)
    g = _generator(seed, 2)
    turn = float(torch.rand(1, generator=g, device="cuda")) * PI
    sx = math.radians(fwhm_deg * math.sqrt((1 + ellipticity) / (1 - ellipticity))) / 2.35482
    sy = math.radians(fwhm_deg * math.sqrt((1 - ellipticity) / (1 + ellipticity))) / 2.35482
    x, y = theta * torch.cos(phi - turn), theta * torch.sin(phi - turn)
    w = torch.exp(-0.5 * ((x / sx) ** 2 + (y / sy) ** 2))
    w = w / (w.sum() * (nside / nside_beam) ** 2)
    leak = 0.01 * w * torch.sin(2.0 * phi)
    small = 0.003 * w * torch.cos(phi)
    a = [(1 + EPSILON) * w, (1 - EPSILON) * w, leak, small]
    b = [(1 + EPSILON) * w, (1 - EPSILON) * w, -leak, small]
    return torch.stack(a + b, dim=1).float().contiguous()


def _scan(kind, n, seed):
    """ra, dec, pa (float64, radians): the sweep (a turn in RA per 4096 samples, 0.05 degrees in Dec
    per sweep), the sweep with every tenth sample within a degree of a pole, or the raster."""
    g = _generator(seed, 3)
    r = [float(v) for v in torch.rand(2, generator=g, device="cuda", dtype=F64)]
    i = torch.arange(n, device="cuda")
    pa = PI * torch.rand(n, generator=g, device="cuda", dtype=F64)
    if kind == "raster":
        cols = -(-n // 121)
        dec = -30.0 + 0.5 * (i // cols) + 0.5 * r[0]
        ra = 60.0 * (i % cols) / max(1, cols - 1) + 360.0 * r[1]
        pa = 0.25 * PI * (i % 4).to(F64)
    else:
        ra = 360.0 * ((i % 4096) + r[0]) / 4096.0
        dec = -80.0 + 130.0 * r[1] + 0.05 * (i // 4096)
    ra, dec = torch.deg2rad(ra.to(F64)), torch.deg2rad(dec.to(F64))
    if kind == "poles":
        at = torch.arange(0, n, 10, device="cuda")
        u = torch.rand((3, at.numel()), generator=g, device="cuda", dtype=F64)
        colat = math.radians(1.0) * torch.sqrt(u[0])
        dec[at] = torch.where(u[1] < 0.5, 0.5 * PI - colat, colat - 0.5 * PI)
        ra[at] = 2.0 * PI * u[2]
    return ra.contiguous(), dec.contiguous(), pa.contiguous()


def _detectors(case, seed):
    """Radius, samples and boresight offset of every pair of a focal plane."""
    r = np.random.default_rng([int(seed), 4])
    nd = case["ndet"]
    radius = r.uniform(1.0, 5.0, nd)
    ell = r.uniform(0.0, 0.1, nd)
    off = np.radians(r.uniform(-1.4, 1.4, (2, nd)))
    # the sample counts are the case's own, whatever the seed
    r = np.random.default_rng([nd, case["most"]])
    n = np.exp(r.uniform(math.log(case["least"]), math.log(case["most"]), nd)).astype(int)
    return [(float(radius[d]), float(ell[d]), int(n[d]), float(off[0, d]), float(off[1, d]))
            for d in range(nd)]


def _detector(case, seed, d, det):
    radius, ell, n, dx, dy = det
    beam = _beam(case["nside"], case["nside_beam"], radius, radius / 2.5, ell, seed + 100 * d)
    ra, dec, pa = _scan("sweep", n, seed + 100 * d)
    dec = dec + dy
    ra = torch.remainder(ra + dx / torch.cos(dec), 2.0 * PI)
    return beam, ra.contiguous(), dec.contiguous(), pa


def _inputs(case, seed):
    sky = _sky(case["nside"], seed)
    beam = _beam(case["nside"], case["nside_beam"], case["radius"], case["radius"] / 2.0, 0.05, seed)
    return sky, beam, _scan(case.get("scan", "sweep"), case["n"], seed)


def _parameters():
    return torch.tensor([1.2, 0.05, 20.0, 2e-4, -1e-4])


def _residuals(case, seed, n):
    g = _generator(seed, 5)
    return [40.0 * torch.randn(n, generator=g, device="cuda") for _ in range(2)]


def _stream():
    return torch.cuda.current_stream().cuda_stream or 1  # 1: the legacy default stream


class _Convolver:
    """A convolver with its sky, beam and scan resident."""

    def __init__(self, case, sky, beam, scan):
        self.conv = GPUConvolver()
        self.conv.set_sky_device(case["nside"], sky.data_ptr(), False, stream=_stream())
        self.conv.set_beam_device(case["nside_beam"], beam.shape[0], beam.data_ptr(), False, stream=_stream())
        self.conv.set_scan_device(case["n"], *[v.data_ptr() for v in scan], stream=_stream())
        torch.cuda.synchronize()


class _Array:
    """A device array of a handle, for torch.as_tensor."""

    def __init__(self, owner, pointer, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=kind, data=(pointer, False), version=3)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "pointing":
        lib = _lib.load()
        st["call"] = lib.pisco_focal_plane_to_sky_device
        st["dets"], st["centre"] = _focal(case, seed)
        st["out"] = [torch.empty((case["ndet"], case["n"]), dtype=F64, device="cuda") for _ in range(3)]
        return st
    if kind == "mapmake":
        st["map"] = SkyMap(case["nside"])
        st["scan"], st["pol"], st["data"] = _binned(case, seed)
        return st
    if kind == "batched":
        conv = GPUConvolver()
        sky = _sky(case["nside"], seed)
        conv.set_sky_device(case["nside"], sky.data_ptr(), False, stream=_stream())
        torch.cuda.synchronize()
        rows, st["keep"], st["tod"] = [], [], []
        for d, det in enumerate(_detectors(case, seed)):
            maps, ra, dec, pa = _detector(case, seed, d, det)
            beam = PolBeam(case["nside_beam"], maps.shape[0], EPSILON, "p")
            host = maps.t().contiguous().cpu().numpy()
            beam.aBeams, beam.bBeams = list(host[:4]), list(host[4:])
            conv.set_beam_slot(d, beam)
            tod = [torch.empty(ra.numel(), device="cuda") for _ in range(2)]
            rows.append((d, ra.numel(), ra.data_ptr(), dec.data_ptr(), pa.data_ptr(),
                         tod[0].data_ptr(), tod[1].data_ptr()))
            st["keep"].append((ra, dec, pa))
            st["tod"].append(tod)
        st["conv"], st["rows"] = conv, conv.det_descs(rows)
        return st
    sky, beam, scan = _inputs(case, seed)
    if kind == "host":
        st["conv"] = conv = GPUConvolver(form=case["form"])
        planes = beam.t().contiguous().cpu().numpy()
        conv.set_beam_planes(case["nside_beam"], beam.shape[0], planes[:4], planes[4:])
        conv.set_sky_device(case["nside"], sky.double().contiguous().data_ptr(), True, stream=_stream())
        torch.cuda.synchronize()
        st["scan"] = [v.cpu().numpy() for v in scan]
        # GPUConvolver's callers hold float32 TOD, as its C++ class does
        kind = np.float64 if case["form"] == "plain" else np.float32
        st["out"] = [np.empty(case["n"], kind) for _ in range(2)]
        return st
    st["conv"] = conv = _Convolver(case, sky, beam, scan).conv
    n = case["n"]
    if kind == "forward":
        conv.set_interp(case["bilinear"])
        conv.set_sample_order(case["order"])
        st["out"] = [torch.empty(n, dtype=F64 if case["form"] == "fp64" else torch.float32, device="cuda")
                     for _ in range(2)]
    elif kind == "adjoint":
        st["g"] = _residuals(case, seed, n)
        st["out"] = torch.empty((12 * case["nside"] ** 2, 4), device="cuda")
    else:
        st["sky"] = sky[:, :3].contiguous().requires_grad_(True)
        st["beam"] = beam.requires_grad_(True) if kind == "maps" else beam
        st["parameters"] = _parameters().requires_grad_(True)
        st["target"] = _residuals(case, seed, n)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "pointing":
        p = [v.data_ptr() for v in st["dets"]]
        c = [v.data_ptr() for v in st["centre"]]
        _lib.check(st["call"](case["ndet"], *p, case["n"], *c, 1, *[v.data_ptr() for v in st["out"]],
                              _stream()), None, "focal_plane_to_sky")
        return st["out"]
    if kind == "mapmake":
        m = st["map"]
        m.reset()
        m.accumulate_device(case["n"], *[v.data_ptr() for v in st["scan"]], case["ndet"], st["pol"],
                            st["data"].data_ptr(), f64=False, stream=_stream())
        m.solve_map()
        iqu, hits, normal = m.device_arrays()
        npix = m.size()
        return dict(iqu=torch.as_tensor(_Array(m, iqu, (3, npix), "<f4"), device="cuda"),
                    hits=torch.as_tensor(_Array(m, hits, (npix,), "<i4"), device="cuda"),
                    normal=torch.as_tensor(_Array(m, normal, (9, npix), "<f8"), device="cuda"))
    conv = st["conv"]
    if kind == "batched":
        conv.forward_batched(st["rows"], stream=_stream())
        return dict(a=torch.cat([t[0] for t in st["tod"]]), b=torch.cat([t[1] for t in st["tod"]]))
    if kind == "host":
        conv.update_scan(Scan(case["n"], *st["scan"]))
        conv.exec_convolution(*st["out"], polFlag="p")
        return st["out"]
    if kind == "forward":
        conv.forward_device(st["out"][0].data_ptr(), st["out"][1].data_ptr(),
                            out_f64=case["form"] == "fp64", stream=_stream(), form=case["form"])
        return st["out"]
    if kind == "adjoint":
        conv.adjoint_device(st["g"][0].data_ptr(), st["g"][1].data_ptr(), False, st["out"].data_ptr(), 0,
                            deterministic=case["deterministic"], stream=_stream())
        return st["out"]
    if kind == "maps":
        tod = convolve(st["sky"], st["beam"], conv, case["nside"], case["nside_beam"])
        leaves = (st["sky"], st["beam"])
    else:
        tod = convolve_gaussian(st["sky"], st["parameters"], conv, case["nside"], case["nside_beam"],
                                st["beam"].shape[0], EPSILON)
        leaves = (st["sky"], st["parameters"])
    loss = sum(0.5 * torch.sum((t - y) ** 2) for t, y in zip(tod, st["target"]))
    grads = torch.autograd.grad(loss, leaves)
    return dict(a=tod[0].detach(), b=tod[1].detach(), sky=grads[0], beam=grads[1])


def work(case):
    kind = case["kind"]
    if kind == "pointing":
        n = case["ndet"] * case["n"]
        return {"bytes": 24 * case["n"] + 24 * case["ndet"] + 24 * n, "flops": 300 * n}
    npix = 12 * case["nside"] ** 2
    if kind == "mapmake":
        n = case["ndet"] * case["n"]
        return {"bytes": 16 * n + 12 * npix + 4 * npix + 72 * npix, "flops": 150 * n + 60 * npix}

    def pairs(radius):
        return npix * (1.0 - math.cos(math.radians(radius))) / 2.0

    def seen(radius, n):
        sweeps = -(-n // 4096)
        lit = min(1.0, (2.0 * radius + 0.05 * sweeps) / 180.0 + (0.01 if n > 4 else 0.0))
        return min(npix * lit, pairs(radius) * n)

    if kind == "batched":
        dets = _detectors(case, 0)
        n = sum(d[2] for d in dets)
        return {"bytes": 16 * max(seen(3.0, d[2]) for d in dets) + 32 * n +
                32 * len(dets) * 6.0 * case["nside_beam"] ** 2 * (1.0 - math.cos(math.radians(3.0))),
                "flops": FLOPS * sum(d[2] for d in dets) * pairs(3.0)}
    r, n = case["radius"], case["n"]
    wide = 2 if case.get("form") == "fp64" else 1
    sky = 16 * wide * seen(r, n)
    beam = 32 * wide * 6.0 * case["nside_beam"] ** 2 * (1.0 - math.cos(math.radians(r)))
    out = (16 if case.get("form") == "fp64" or kind == "host" and case["form"] == "plain" else 8) * n
    flops = FLOPS * n * pairs(r) * (2.0 if case.get("bilinear") else 1.0)
    if kind == "adjoint":
        return {"bytes": beam + 32 * n + 16 * npix, "flops": flops}
    if kind == "maps":
        return {"bytes": 12 * npix * 2 + 2 * beam + 40 * n, "flops": 2.2 * flops}
    if kind == "params":
        return {"bytes": 12 * npix * 2 + beam + 40 * n, "flops": 2.2 * flops}
    return {"bytes": sky + beam + 24 * n + out, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch
def _focal(case, seed):
    g = _generator(seed, 6)
    nd, n = case["ndet"], case["n"]
    dets = [math.radians(15.0) * (torch.rand(nd, generator=g, device="cuda", dtype=F64) - 0.5) for _ in range(2)]
    dets.append(PI * torch.rand(nd, generator=g, device="cuda", dtype=F64))
    ra, dec, pa = _scan("sweep", n, seed)
    return dets, [ra, 0.9 * dec, 0.5 * pa]


def _binned(case, seed):
    """Pointing of ndet detectors (the same boresight, as a focal-plane pixel has), their angles and
    TOD, det-major float32."""
    g = _generator(seed, 7)
    nd, n = case["ndet"], case["n"]
    ra, dec, pa = _scan("sweep", n, seed)
    # neighbouring sweeps, so that pixels are hit by several of them
    dec = dec + math.radians(0.2) * torch.rand(n, generator=g, device="cuda", dtype=F64)
    scan = [v.float().repeat(nd).contiguous() for v in (ra, dec, pa)]
    pol = (np.arange(nd) * (PI / nd)).astype(np.float32)
    return scan, pol, 100.0 * torch.randn(nd * n, generator=g, device="cuda")


def _pairs(nside, rho_max, ra, dec):
    """Sample, ring and pixel of every disc pixel of the samples (HEALPix query_disc)."""
    z, count, shift, start = _rings(nside)
    th = 0.5 * PI - dec
    z0, s0 = torch.cos(th), torch.sin(th)

    def above(x):
        eq = (nside * (2.0 - 1.5 * x)).long()
        cap = (nside * torch.sqrt(3.0 * (1.0 - x.abs()))).long()
        return torch.where(x.abs() <= 2.0 / 3.0, eq, torch.where(x > 0, cap, 4 * nside - cap - 1))

    lo = above(torch.cos(th - rho_max)) + 1
    hi = above(torch.cos(th + rho_max))
    first = torch.where(th - rho_max <= 0, torch.ones_like(lo), lo)
    last = torch.where(th + rho_max >= PI, torch.full_like(hi, 4 * nside - 1), hi)
    rows = last - first + 1
    smp = torch.repeat_interleave(torch.arange(ra.numel(), device="cuda"), rows)
    ring = torch.arange(smp.numel(), device="cuda") - (torch.cumsum(rows, 0) - rows)[smp] + first[smp]
    i = ring - 1
    x = (math.cos(rho_max) - z[i] * z0[smp]) / s0[smp]
    ysq = 1.0 - z[i] ** 2 - x * x
    half = torch.where(ysq > 0, torch.atan2(torch.sqrt(ysq.clamp(min=0)), x), torch.zeros_like(x))
    fr = count[i].to(F64) / (2.0 * PI)
    a = torch.floor(fr * (ra[smp] - half) - shift[i]).long() + 1
    b = torch.floor(fr * (ra[smp] + half) - shift[i]).long()
    whole = (ring < lo[smp]) | (ring > hi[smp])
    a = torch.where(whole, torch.zeros_like(a), a)
    num = torch.where(whole, count[i], torch.where(half > 0, b - a + 1, torch.zeros_like(a))).clamp(min=0)
    seg = torch.repeat_interleave(torch.arange(num.numel(), device="cuda"), num)
    j = torch.arange(seg.numel(), device="cuda") - (torch.cumsum(num, 0) - num)[seg] + a[seg]
    i = i[seg]
    phi = (j.to(F64) + shift[i]) * (2.0 * PI / count[i].to(F64))
    return smp[seg], z[i], phi, start[i] + torch.remainder(j, count[i])


def _geometry(zp, phi, ra, dec, pa):
    """1 - cos(rho), rho, sigma in [0, 2 pi) and cos, sin of 2 chi of pixels seen from their samples."""
    psi = -pa
    sp = torch.sqrt((1.0 - zp) * (1.0 + zp))
    s0, c0 = torch.sin(dec), torch.cos(dec)
    d = phi - ra
    sd, cd = torch.sin(d), torch.cos(d)
    q = 2.0 * torch.sin(0.5 * (torch.asin(zp) - dec)) ** 2 + 2.0 * sp * c0 * torch.sin(0.5 * d) ** 2
    u, v = sp * sd, zp * c0 - sp * s0 * cd
    nb, db = c0 * sd, s0 * sp - c0 * zp * cd
    rho = 2.0 * torch.asin(torch.sqrt(0.5 * q))
    tiny = rho <= 1e-6
    al = torch.where(tiny, torch.full_like(u, 0.5 * PI), torch.atan2(u, v))
    be = torch.where(tiny, torch.full_like(u, 0.5 * PI), torch.atan2(nb, db))
    sig = torch.remainder(PI - al - psi, 2.0 * PI)
    chi = be - (PI - al - psi)
    return q, rho, sig, torch.cos(2.0 * chi), torch.sin(2.0 * chi)


def _stencil(nside_beam, npix, q, rho, sig, bilinear):
    """Beam pixels and weights of every pair: pixel columns (-1: outside) with weights that sum to 1."""
    r = nside_beam * torch.sqrt(3.0 * q)
    if not bilinear:
        tt = torch.remainder(sig * (2.0 / PI), 4.0)
        tp = tt - torch.floor(tt)
        ir = torch.floor(tp * r).long() + torch.floor((1.0 - tp) * r).long() + 1
        px = 2 * ir * (ir - 1) + torch.floor(tt * ir.to(F64)).long()
        return [torch.where(px < npix, px, torch.full_like(px, -1))], [(px < npix).to(F64)]
    k = torch.floor(r).long()

    def colat(i):
        return 2.0 * torch.asin(i.to(F64) / (math.sqrt(6.0) * nside_beam))

    def on(i):
        t = sig * (4.0 * i.to(F64)) / (2.0 * PI) - 0.5
        f = torch.floor(t)
        w = t - f
        a = f.long()
        first = 2 * i * (i - 1)
        return first + torch.remainder(a, 4 * i), first + torch.remainder(a + 1, 4 * i), 1.0 - w, w

    cap = k == 0
    kk = torch.where(cap, torch.ones_like(k), k)
    p1, p2, w1, w2 = on(kk)
    p3, p4, w3, w4 = on(k + 1)
    wt = (rho - colat(k)) / (colat(k + 1) - colat(k))
    f = 0.25 * (1.0 - wt)
    px = [torch.where(cap, (p3 + 2) & 3, p1), torch.where(cap, (p4 + 2) & 3, p2), p3, p4]
    ws = [torch.where(cap, f, w1 * (1.0 - wt)), torch.where(cap, f, w2 * (1.0 - wt)),
          w3 * wt + torch.where(cap, f, torch.zeros_like(f)), w4 * wt + torch.where(cap, f, torch.zeros_like(f))]
    ws = [torch.where(p < npix, w, torch.zeros_like(w)) for p, w in zip(px, ws)]
    total = ws[0] + ws[1] + ws[2] + ws[3]
    ws = [torch.where(total > 0, w / total.clamp(min=1e-300), torch.zeros_like(w)) for w in ws]
    return [torch.where(p < npix, p, torch.full_like(p, -1)) for p in px], ws


def _rho_max(nside_beam, npix):
    i = int(round((1.0 + math.sqrt(1.0 + 2.0 * npix)) / 2.0))
    t = i * i / (3.0 * nside_beam * nside_beam)
    return math.atan2(math.sqrt(t * (2.0 - t)), 1.0 - t)


def _walk(nside, nside_beam, npix, scan, bilinear, f):
    """f(first, end, sample, sky pixel, beam pixels, weights, cos 2 chi, sin 2 chi) over the scan in parts."""
    ra, dec, pa = scan
    rho_max = _rho_max(nside_beam, npix)
    per = max(1.0, 6.0 * nside * nside * (1.0 - math.cos(rho_max)))
    step = max(1, int(1.5e7 / per))
    for at in range(0, ra.numel(), step):
        end = min(ra.numel(), at + step)
        r, d, p = ra[at:end], dec[at:end], pa[at:end]
        smp, zp, phi, sky_pixel = _pairs(nside, rho_max, r, d)
        q, rho, sig, c2, s2 = _geometry(zp, phi, r[smp], d[smp], p[smp])
        px, ws = _stencil(nside_beam, npix, q, rho, sig, bilinear)
        f(at, end, smp, sky_pixel, px, ws, c2, s2)


def _value(maps, px, ws):
    out = torch.zeros((px[0].numel(), maps.shape[1]), dtype=F64, device="cuda")
    for p, w in zip(px, ws):
        out += maps[p.clamp(min=0)] * w[:, None]
    return out


def _tod(case, sky, beam, scan, bilinear=False):
    sky, beam = sky.double(), beam.double()
    out = torch.zeros((2, scan[0].numel()), dtype=F64, device="cuda")

    def part(at, end, smp, sp, px, ws, c2, s2):
        s, b = sky[sp], _value(beam, px, ws)
        qr, ur = s[:, 1] * c2 + s[:, 2] * s2, s[:, 2] * c2 - s[:, 1] * s2
        out[0, at:end].index_add_(0, smp, s[:, 0] * b[:, 0] + qr * b[:, 1] + ur * b[:, 2] + s[:, 3] * b[:, 3])
        out[1, at:end].index_add_(0, smp, s[:, 0] * b[:, 4] - qr * b[:, 5] - ur * b[:, 6] + s[:, 3] * b[:, 7])

    _walk(case["nside"], case["nside_beam"], beam.shape[0], scan, bilinear, part)
    return out


def _transpose(case, sky, beam, scan, ga, gb):
    sky, beam = sky.double(), beam.double()
    gs, gm = torch.zeros_like(sky), torch.zeros_like(beam)

    def part(at, end, smp, sp, px, ws, c2, s2):
        wa, wb = ga[at:end][smp], gb[at:end][smp]
        s, b = sky[sp], _value(beam, px, ws)
        q, u = wa * b[:, 1] - wb * b[:, 5], wa * b[:, 2] - wb * b[:, 6]
        gs.index_add_(0, sp, torch.stack([wa * b[:, 0] + wb * b[:, 4], q * c2 - u * s2, q * s2 + u * c2,
                                          wa * b[:, 3] + wb * b[:, 7]], dim=1))
        qr, ur = s[:, 1] * c2 + s[:, 2] * s2, s[:, 2] * c2 - s[:, 1] * s2
        g = torch.stack([wa * s[:, 0], wa * qr, wa * ur, wa * s[:, 3],
                         wb * s[:, 0], -wb * qr, -wb * ur, wb * s[:, 3]], dim=1)
        for p, w in zip(px, ws):
            gm.index_add_(0, p.clamp(min=0), g * w[:, None])

    _walk(case["nside"], case["nside_beam"], beam.shape[0], scan, False, part)
    return gs, gm


def _model(case, p):
    """npix x 8 beam maps of the elliptical Gaussian pair of p, differentiable."""
    npix, theta, phi = _beam_pixels(case["nside_beam"], case["radius"])
    fwhm, e, turn, dx, dy = p
    d2r = PI / 180.0
    sx = d2r * fwhm * torch.sqrt((1 + e) / (1 - e)) / 2.35482
    sy = d2r * fwhm * torch.sqrt((1 - e) / (1 + e)) / 2.35482
    t = d2r * turn
    ca = torch.cos(t) ** 2 / (2 * sx * sx) + torch.sin(t) ** 2 / (2 * sy * sy)
    cb = -torch.sin(2 * t) / (4 * sx * sx) + torch.sin(2 * t) / (4 * sy * sy)
    cc = torch.sin(t) ** 2 / (2 * sx * sx) + torch.cos(t) ** 2 / (2 * sy * sy)
    x, y = theta * torch.cos(phi) - dx, theta * torch.sin(phi) - dy
    g = torch.exp(-(ca * x * x + 2.0 * cb * x * y + cc * y * y))
    g = g / (g.sum() * (case["nside"] / case["nside_beam"]) ** 2)
    z = torch.zeros_like(g)
    a = torch.stack([(1 + EPSILON) * g, (1 - EPSILON) * g, z, z], dim=1)
    return torch.cat([a, a], dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pointing":
        (dx, dy, pol), (x, y, rot) = _focal(case, seed)
        dx, dy, pol = dx[:, None], dy[:, None], pol[:, None]
        cr = torch.cos(dx) * torch.cos(dy)
        sr = torch.sqrt((1.0 - cr) * (1.0 + cr))
        g = 0.5 * PI - torch.atan2(torch.sin(dy), torch.sin(dx) * torch.cos(dy)) - rot
        sl, cl, se, ce = torch.sin(y), torch.cos(y), torch.sin(rot), torch.cos(rot)
        lat = torch.asin(cr * sl + sr * cl * torch.cos(g))
        pa = torch.atan2(cl * se * torch.cos(dx) - sl * torch.sin(dx),
                         cl * ce * torch.cos(dy) - (sl * torch.cos(dx) + cl * se * torch.sin(dx)) * torch.sin(dy))
        lon = x - torch.atan2(sr * torch.sin(g), cr * cl - sr * sl * torch.cos(g))
        return [lon, lat, pa + pol]
    if kind == "mapmake":
        return _exact_maps(case, seed)
    if kind == "batched":
        sky = _sky(case["nside"], seed)
        got = []
        for d, det in enumerate(_detectors(case, seed)):
            beam, *scan = _detector(case, seed, d, det)
            got.append(_tod(case, sky, beam, scan))
        return dict(a=torch.cat([g[0] for g in got]), b=torch.cat([g[1] for g in got]))
    sky, beam, scan = _inputs(case, seed)
    if kind == "host":
        return [v.cpu().numpy() for v in _tod(case, sky, beam, scan)]
    if kind == "forward":
        return list(_tod(case, sky, beam, scan, case["bilinear"]))
    if kind == "adjoint":
        ga, gb = [g.double() for g in _residuals(case, seed, case["n"])]
        return _transpose(case, sky, beam, scan, ga, gb)[0]
    target = [t.double() for t in _residuals(case, seed, case["n"])]
    p = None
    if kind == "params":
        p = _parameters().to("cuda", F64).requires_grad_(True)
        beam = _model(case, p)
    tod = _tod(case, sky, beam.detach(), scan)
    gs, gm = _transpose(case, sky, beam.detach(), scan, tod[0] - target[0], tod[1] - target[1])
    if p is not None:
        gm = torch.autograd.grad(beam, p, gm)[0]
    return dict(a=tod[0], b=tod[1], sky=gs[:, :3].contiguous(), beam=gm)


def _exact_maps(case, seed):
    (ra, dec, pa), pol, data = _binned(case, seed)
    nside, npix = case["nside"], 12 * case["nside"] ** 2
    ra, dec, pa, data = [v.double() for v in (ra, dec, pa, data)]
    psi = -(torch.as_tensor(pol, device="cuda").double().repeat_interleave(case["n"]) + pa)
    z = torch.cos(0.5 * PI - dec)
    tt = torch.remainder(ra * (2.0 / PI), 4.0)
    t1, t2 = nside * (0.5 + tt), nside * z * 0.75
    jp, jm = torch.floor(t1 - t2).long(), torch.floor(t1 + t2).long()
    ir = nside + 1 + jp - jm
    ip = torch.remainder((jp + jm - nside + (1 - (ir & 1)) + 1) // 2, 4 * nside)
    equator = 2 * nside * (nside - 1) + (ir - 1) * 4 * nside + ip
    r = nside * torch.sqrt(3.0 * (1.0 - z.abs()))
    tp = tt - torch.floor(tt)
    ir = torch.floor(tp * r).long() + torch.floor((1.0 - tp) * r).long() + 1
    ip = torch.floor(tt * ir.to(F64)).long()
    cap = torch.where(z > 0, 2 * ir * (ir - 1) + ip, npix - 2 * ir * (ir + 1) + ip)
    pix = torch.where(z.abs() <= 2.0 / 3.0, equator, cap)
    c, s = torch.cos(2.0 * psi), torch.sin(2.0 * psi)
    one = torch.ones_like(c)
    normal = torch.zeros((9, npix), dtype=F64, device="cuda")
    for k, v in enumerate((one, c, s, c * c, c * s, s * s, data, c * data, s * data)):
        normal[k].index_add_(0, pix, v)
    n, sc, ss, cc, cs, s2, d, cd, sd = normal
    hits = n.long()
    at = torch.nonzero(hits >= 3)[:, 0]
    a = torch.stack([n, sc, ss, sc, cc, cs, ss, cs, s2])[:, at].t().reshape(-1, 3, 3)
    iqu = torch.zeros((3, npix), dtype=F64, device="cuda")
    iqu[:, at] = torch.linalg.solve(a, torch.stack([d, cd, sd], dim=1)[at]).t()
    return dict(iqu=iqu, hits=None, normal=normal)
