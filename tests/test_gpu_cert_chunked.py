"""The chunked certified kernels (csrc/cert_point.cuh) against the general
certified kernels, over the forms of calls they take: projections,
pixelizors, components, timeline lengths around the 64-sample chunks, sample
ranges that start anywhere, detector weights, unaligned rows, smooth,
jittering and rough boresights, and odd values.  Every term must be the
general path's: from_map bit for bit, to_map and to_weight_map up to the
order of the float64 additions (each pixel's sum of a few thousand terms at
most is within 1e-12 of the map's largest value)."""
import numpy as np
import pytest

import so3g_gb300
from so3g_gb300 import _abi, synth
from so3g_gb300.proj import quat
from so3g_gb300.proj.ranges import RangesMatrix
from so3g_gb300.proj.wcs import ProjectionistHealpix
from conftest import bits_equal

pytestmark = pytest.mark.gpu

GEOMS = ["CAR", "CAR-tiled", "TAN", "TAN-tiled", "ZEA", "SIN", "HP-RING", "HP-NEST", "HP-tiled"]


def _projectionist(geom, el):
    kind, _, opt = geom.partition("-")
    if kind == "HP":
        if opt == "tiled":
            return ProjectionistHealpix.for_healpix(512, nside_tile=8, active_tiles=range(768),
                                                    ordering="NEST")
        return ProjectionistHealpix.for_healpix(512, ordering=opt)
    return synth.car_projectionist((301, 407), 2 * synth.ARCMIN, el=el, proj=kind,
                                   tile_shape=(64, 96) if opt else None)


def _inputs(geom, n_det, n_time, t0=0., noise=0., el=50., throw=4.):
    import torch
    rng = np.random.default_rng(n_time + n_det)
    p = _projectionist(geom, el)
    dets, resp, _ = synth.focal_plane(rng, n_det, 1.5)
    resp = np.stack([np.ones(n_det), rng.uniform(0.5, 1.1, n_det)], 1).astype(np.float32)
    Q, _ = synth.scan(n_time, el=el, throw=throw, t0=t0)
    q = synth.native(p, Q)
    if noise:
        q = q + noise * rng.standard_normal(q.shape)
        q /= np.sqrt((q * q).sum(1, keepdims=True))
    return p, [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (q, dets, resp)], rng


def _both(call):
    """call() with the chunked kernels and with the general ones."""
    out = []
    for least in (0, 1 << 62):
        so3g_gb300.set_chunked_min_samples(least)
        out.append(call())
    so3g_gb300.set_chunked_min_samples(0)
    return out


def _flat(m):
    m = m if isinstance(m, list) else [m]
    return np.concatenate([x.cpu().numpy().ravel() for x in m if x is not None])


def _maps_close(pair):
    a, b = (_flat(m) for m in pair)
    ok = np.isfinite(b)
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[~ok & ~np.isnan(b)], b[~ok & ~np.isnan(b)])
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * max(np.abs(b[ok]).max(), 1e-300)
    assert (b != 0).any()


def _check_all(eng, args, rng, weights=None, ranges=None, stride=0, sig=None):
    import torch
    n_time, n_det = args[0].shape[0], args[1].shape[0]
    if sig is None:
        sig = rng.standard_normal((n_det, n_time)).astype(np.float32)
    buf = torch.zeros((n_det, n_time + stride), dtype=torch.float32, device="cuda")
    s = buf[:, :n_time]
    s.copy_(torch.from_numpy(sig))
    nc = eng.comp_count
    for acc in (None, _abi.ACCUM_ATOMIC):
        _maps_close(_both(lambda: eng.to_map(eng.zeros(nc, device="cuda"), *args, s, weights,
                                             ranges, accum=acc)))
    _maps_close(_both(lambda: eng.to_weight_map(eng.zeros((nc, nc), device="cuda"), *args, weights,
                                                ranges)))
    m = eng.zeros(nc, device="cuda")
    for t in (m if isinstance(m, list) else [m]):
        t.copy_(torch.from_numpy(rng.standard_normal(tuple(t.shape))))
        t.flatten()[::7] = 0.0
        t.flatten()[3::7] = -0.0

    def scan():
        out = s.clone()
        return eng.from_map(m, *args, out)

    a, b = (x.cpu().numpy() for x in _both(scan))
    assert bits_equal(a, b)


@pytest.mark.parametrize("comps", ["T", "QU", "TQU"])
@pytest.mark.parametrize("geom", GEOMS)
def test_geometries(gpulib, geom, comps):
    """Smooth boresight: the quartic models."""
    p, args, rng = _inputs(geom, 5, 3000, el=45.)
    _check_all(p.get_ProjEng(comps), args, rng)


@pytest.mark.parametrize("comps", ["T", "QU", "TQU"])
@pytest.mark.parametrize("geom", ["CAR", "CAR-tiled", "HP-NEST"])
def test_from_map_onto_zeros(gpulib, geom, comps):
    """Sums that are exact zeros of either sign, subnormal or tiny: a third
    of the map zero, rows that start from +-0 and at the end of float32's
    range, a detector without polarisation response."""
    import torch
    p, args, rng = _inputs(geom, 6, 3003, el=45.)
    args[2][2, 1] = 0.0
    eng = p.get_ProjEng(comps)
    m = eng.zeros(eng.comp_count, device="cuda")
    for t in (m if isinstance(m, list) else [m]):
        x = rng.standard_normal(tuple(t.shape)) * 10. ** rng.integers(-42, 2, tuple(t.shape))
        x[rng.random(tuple(t.shape)) < 0.2] = 0.0
        x[rng.random(tuple(t.shape)) < 0.2] = -0.0
        t.copy_(torch.from_numpy(x))
    sig = torch.zeros((6, 3003), dtype=torch.float32, device="cuda")
    sig[1::3] = -0.0
    sig[5] = 1e-39
    a, b = (x.cpu().numpy() for x in _both(lambda: eng.from_map(m, *args, sig.clone())))
    assert (b != 0).any() and bits_equal(a, b)


@pytest.mark.parametrize("n_time", [64, 65, 66, 127, 128, 129, 2048, 2049, 16385])
def test_timeline_lengths(gpulib, n_time):
    """Around chunks (64), groups (2048) and pieces (16384); 64 samples do
    not make a model."""
    p, args, rng = _inputs("CAR", 3, n_time)
    _check_all(p.get_ProjEng("TQU"), args, rng, stride=1)


@pytest.mark.parametrize("geom", ["CAR", "ZEA", "HP-RING"])
@pytest.mark.parametrize("t0,noise", [(1.7e9, 0.), (0., 1e-9), (0., 1e-8), (0., 1e-7), (0., 1e-5)])
def test_rough_boresight(gpulib, geom, t0, noise):
    """Time-stamp jitter and pointing noise: quadratic models with
    residuals, and boresights left to the general kernel."""
    p, args, rng = _inputs(geom, 4, 5000, t0=t0, noise=noise)
    _check_all(p.get_ProjEng("TQU"), args, rng)


@pytest.mark.parametrize("comps", ["T", "TQU"])
@pytest.mark.parametrize("geom", ["CAR", "ZEA", "HP-RING"])
@pytest.mark.parametrize("n_time", [4449, 4481])
def test_turn_arounds_everywhere(gpulib, geom, comps, n_time):
    """A turn-around every 67 samples: at every offset within a chunk, and in
    the last chunk, of one sample or of 33."""
    p, args, rng = _inputs(geom, 4, n_time, el=45., throw=67 / 200.)
    _check_all(p.get_ProjEng(comps), args, rng)


@pytest.mark.parametrize("geom", ["CAR", "CAR-tiled"])
def test_ranges_and_weights(gpulib, geom):
    """Ranges starting and ending anywhere, overlapping, some empty."""
    import torch
    p, args, rng = _inputs(geom, 6, 4003)
    w = torch.from_numpy(np.array([1., 0., 0.3, 2., 1.5, 1e-3], np.float32)).cuda()
    mask = rng.random((6, 4003)) < 0.995
    mask[2] = False
    mask[4, 100:163] = False
    one = RangesMatrix.from_mask(mask)
    two = RangesMatrix.from_mask(rng.random((6, 4003)) < 0.5)
    for r in (one, [one, two], RangesMatrix.from_mask(torch.from_numpy(mask).cuda())):
        _check_all(p.get_ProjEng("TQU"), args, rng, weights=w, ranges=r)


def test_odd_values(gpulib):
    """Infinite, NaN and huge signals, a response of zero, a quaternion that
    is NaN and one that is not of unit length."""
    p, args, rng = _inputs("CAR", 4, 3000)
    sig = rng.standard_normal((4, 3000)).astype(np.float32)
    sig[0, 100], sig[1, 200], sig[2, 300:340], sig[3, 700] = np.inf, np.nan, 3e38, -np.inf
    sig[0, 1000:1100] = 1e-44
    args[2][1, 1] = 0.
    args[2][2, 1] = -0.75
    _check_all(p.get_ProjEng("TQU"), args, rng, sig=sig)
    args[0][1500] = float("nan")
    args[0][2000:2050] *= 1.0001
    _check_all(p.get_ProjEng("TQU"), args, rng)


def test_seam_pole_and_map_edge(gpulib):
    """A CAR map whose seam and native pole the scan crosses (the models do
    not apply there)."""
    import torch
    q = quat.euler(2, np.linspace(np.pi - 0.05, np.pi + 0.05, 4000)) * quat.euler(
        1, np.linspace(0.01, 1.2, 4000))
    rng = np.random.default_rng(1)
    dets, resp, _ = synth.focal_plane(rng, 4, 1.0)
    p = synth.car_projectionist((440, 880), 25 * synth.ARCMIN, el=0., az0=0.)
    args = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
            for x in (np.asarray(q, dtype=np.float64), dets, resp)]
    _check_all(p.get_ProjEng("TQU"), args, rng)


@pytest.mark.parametrize("mode", [_abi.POINTING_MIXED, _abi.POINTING_CERTIFIED])
@pytest.mark.parametrize("proj,comps", [("ZEA", "TQU"), ("ZEA", "T"), ("TAN", "QU"), ("SIN", "TQU")])
@pytest.mark.parametrize("n_time,t0,noise", [(3001, 0., 0.), (65, 0., 0.), (4099, 1.7e9, 0.),
                                             (5000, 0., 1e-8), (5000, 0., 1e-5)])
def test_bilinear_from_map(gpulib, proj, comps, n_time, t0, noise, mode):
    """from_map of bilinear zenithal maps: the chunked kernels' weights are
    the general kernels' or (a coordinate within 2.5e-7 of a pixel of
    theirs) close to them: 12 products of a map value below |m|, of weights
    off by at most 2 x 2.5e-7 + 2^-23, and, as nearly all weights are the
    same floats, within the rounding of a 12-term float32 sum in the mean."""
    import torch
    p, args, rng = _inputs("ZEA", 5, n_time, t0=t0, noise=noise)
    p = synth.car_projectionist((301, 407), synth.ARCMIN, proj=proj, interpol="bilinear")
    eng = p.get_ProjEng(comps)
    eng.pointing = mode
    m = torch.from_numpy(rng.standard_normal((eng.comp_count, 301, 407))).cuda()
    m[:, ::5, ::7] = 0.
    sig = torch.from_numpy(rng.standard_normal((5, n_time + 1)).astype(np.float32)).cuda()[:, 1:]

    def scan():
        out = sig.clone() if n_time % 2 else sig
        s0 = out.clone()
        eng.from_map(m, *args, out)
        d = out.cpu().numpy().copy()
        out.copy_(s0)
        return d

    a, b = _both(scan)
    assert (b != sig.cpu().numpy()).mean() > 0.05
    d = np.abs(a.astype(np.float64) - b)
    assert d.max() <= 12 * float(m.abs().max()) * 6.2e-7 + 12 * 2.0**-24 * np.abs(b).max()
    assert np.sqrt((d**2).mean()) <= np.sqrt(12) * 2.0**-24 * np.sqrt((b.astype(float)**2).mean())
