"""Performance cases of so3g_gb300: what a map-making program has it do.

Each case is one pass through the public entry points: the ProjEng_*
classes on CUDA tensors, the Projectionist on numpy arrays, and the
differentiable from_map.  The observations are constant-elevation scans
(triangle-wave azimuth, 200 samples per second) of a circular focal plane
over a map centred on the scan, with the sizes of this repository's
workloads (64 detectors x 100k samples up to 1000 x 1M) and the ranges
around them.

listed() holds the cases, draw() gives more of the same ranges, prepare()
makes what a program has in hand before the call, run() is one pass,
work() what the path cannot do without, and exact() the same results in
float64 from plain torch.

Fields of a case:
  op       step (to_map then from_map of its map), to_map, from_map, weights
           (to_weight_map), grad (differentiable from_map, forward and
           backward), precomp (to_map and from_map of stored pointing)
  proj     CAR, ZEA, TAN or HP (HEALPix)
  comps    T, QU or TQU
  mode     default (the pointing an engine starts with) or mixed
  n_det, n_time; ny, nx, res (arcmin) or nside, nest; radius (deg, focal
  plane); el, throw (deg), speed (deg/s) of the scan
  tile     tile side in pixels (flat) or nside_tile (HEALPix), 0: untiled
  bilinear, host (numpy arrays through the Projectionist), cuts (flagged
  samples left out through thread_intervals), det_weights
"""
import math

import numpy as np
import torch

import so3g_gb300 as so3g
from so3g_gb300 import _abi, autograd
from so3g_gb300.proj import coords as proj_coords
from so3g_gb300.proj import quat as proj_quat
from so3g_gb300.proj.geometry import SimpleWCS
from so3g_gb300.proj.ranges import RangesMatrix
from so3g_gb300.proj.wcs import Projectionist

DEG = math.pi / 180
ARCMIN = DEG / 60
RATE = 200.          # samples per second
AZ0 = 180.           # scan centre, degrees
NCOMP = {"T": 1, "QU": 2, "TQU": 3}

_BASE = dict(op="step", proj="CAR", comps="TQU", mode="default", n_det=64, n_time=100_000,
             ny=600, nx=600, res=1.0, nside=0, nest=False, tile=0, radius=1.0, el=50.,
             throw=10., speed=1., bilinear=False, host=False, cuts=False, det_weights=False)


def _case(**kw):
    return dict(_BASE, **kw)


def listed():
    big = dict(n_det=1000, n_time=1_000_000, ny=2000, nx=2000, radius=1.5)
    return [
        # A wafer's worth of quick-look data: launches and call overhead.
        _case(name="car_step_16x4k", n_det=16, n_time=4096, ny=120, nx=160, res=6.0, throw=4.),
        # The smallest configured workload, one solver step on device arrays.
        _case(name="car_step_64x100k"),
        # The same sizes as a so3g user calls it: numpy in, numpy out.
        _case(name="car_host_step_64x100k", host=True),
        # A whole observation into a map with the pointing engines start with.
        _case(name="car_to_map_1000x1M", op="to_map", **big),
        # Scanning a simulated or estimated map back into detector timestreams.
        _case(name="car_from_map_1000x1M", op="from_map", **big),
        # The weight map of an observation, with inverse-variance weights.
        _case(name="car_weights_500x500k", op="weights", det_weights=True,
              **dict(big, n_det=500, n_time=500_000)),
        # A tiled map, ragged sizes, glitch cuts, detector weights.
        _case(name="car_tiled_cuts_301x400k", op="to_map", n_det=301, n_time=400_037, ny=2000,
              nx=2000, radius=1.5, tile=100, cuts=True, det_weights=True),
        # One conjugate-gradient step of a map-maker in mixed pointing.
        _case(name="car_mixed_step_1000x1M", mode="mixed", **big),
        # A wide fast scan into a HEALPix map, and back.
        _case(name="hp_step_400x500k", proj="HP", nside=1024, n_det=400, n_time=500_000,
              radius=1.5, el=45., throw=30., speed=2.),
        # Zenithal map, two components, odd sizes: small-aperture maps.
        _case(name="zea_qu_step_301x200k", proj="ZEA", comps="QU", n_det=301, n_time=200_003,
              ny=1500, nx=1501, res=1.0, radius=1.5),
        # Gradient of a loss of the bilinear scan of a map (forward, backward).
        _case(name="zea_bilinear_grad_400x300k", op="grad", proj="ZEA", bilinear=True, mode="mixed",
              n_det=400, n_time=300_000, ny=3000, nx=3000, res=0.5, radius=1.5),
        # Stored pointing, used at every iteration of a solver.
        _case(name="precomp_step_600x500k", op="precomp", n_det=600, n_time=500_000, ny=2000,
              nx=2000, radius=1.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["step", "step", "to_map", "from_map", "weights", "grad", "precomp"])
    proj = rng.choice(["CAR", "CAR", "CAR", "HP", "ZEA", "TAN"])
    if op == "grad" and proj == "HP":
        proj = "ZEA"
    if op == "precomp":
        proj = "CAR"
    comps = rng.choice(["T", "QU", "TQU", "TQU", "TQU"])
    n_det = _log_int(rng, 16, 1000)
    n_time = _log_int(rng, 4096, max(8192, min(1_000_000, int(1.5e8 // n_det))))
    c = _case(op=op, proj=proj, comps=comps, n_det=n_det, n_time=n_time,
              mode=rng.choice(["default", "default", "mixed"]),
              radius=round(rng.uniform(0.3, 1.8), 3), el=rng.choice([40., 45., 50., 60.]),
              throw=round(rng.uniform(4., 20.), 2), speed=round(rng.uniform(0.5, 2.), 3))
    if proj == "HP":
        c.update(nside=rng.choice([256, 512, 1024, 2048]), nest=rng.random() < 0.5)
        if c["nest"] and rng.random() < 0.5:
            c["tile"] = rng.choice([4, 8, 16])
    else:
        c.update(res=rng.choice([0.5, 1.0, 2.0]), ny=rng.randint(300, 2000),
                 nx=rng.randint(400, 2500), bilinear=op == "grad" or
                 (op != "precomp" and proj == "ZEA" and rng.random() < 0.3))
        if op not in ("grad", "precomp") and rng.random() < 0.25:
            c["tile"] = rng.choice([64, 100, 256])
    if op in ("to_map", "weights"):
        c["det_weights"] = rng.random() < 0.5
        c["cuts"] = rng.random() < 0.4
    elif op == "step" and n_det * n_time < 8_000_000 and not c["tile"] and proj != "HP":
        c["host"] = rng.random() < 0.3
    return c


# ---------------------------------------------------------------------------
# Inputs.

def _qmul(p, q):
    a, b, c, d = p.unbind(-1)
    e, f, g, h = q.unbind(-1)
    return torch.stack([a * e - b * f - c * g - d * h, a * f + b * e + c * h - d * g,
                        a * g - b * h + c * e + d * f, a * h + b * g - c * f + d * e], -1)


def _rz(x):
    o = torch.zeros_like(x)
    return torch.stack([torch.cos(x / 2), o, o, torch.sin(x / 2)], -1)


def _ry(x):
    o = torch.zeros_like(x)
    return torch.stack([torch.cos(x / 2), o, torch.sin(x / 2), o], -1)


def _native_rotation(c, dev):
    """Celestial to native: the map is centred on the scan (lon -AZ0, lat el)."""
    f = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    spin = _rz(f(AZ0 * DEG))
    if c["proj"] == "HP":
        return f([1., 0., 0., 0.])
    if c["proj"] == "CAR":
        return _qmul(_ry(f(c["el"] * DEG)), spin)
    return _qmul(_rz(f(math.pi)), _qmul(_ry(f((c["el"] - 90.) * DEG)), spin))


def _observation(c, seed, dev):
    """Boresight (celestial frame), detector quaternions, responses and
    weights of a seeded observation."""
    g = torch.Generator(device=dev).manual_seed(seed)
    r = lambda *s: torch.rand(*s, dtype=torch.float64, device=dev, generator=g)  # noqa: E731
    period = 4 * c["throw"] / c["speed"]
    t = torch.arange(c["n_time"], dtype=torch.float64, device=dev) / RATE
    phase = ((t + period * r(1)) * c["speed"]) % (4 * c["throw"])
    az = torch.where(phase > 2 * c["throw"], 4 * c["throw"] - phase, phase) - c["throw"] + AZ0
    el = torch.full_like(az, math.pi / 2 - c["el"] * DEG)
    bore = _qmul(_rz(-az * DEG), _ry(el))
    n = c["n_det"]
    k = torch.arange(n, dtype=torch.float64, device=dev)
    rad = c["radius"] * DEG * torch.sqrt((k + 0.5) / n)
    phi = k * (math.pi * (3 - math.sqrt(5.)))
    gamma = math.pi * r(n)
    dets = _qmul(_qmul(_rz(phi), _ry(rad)), _rz(gamma - phi))
    resp = torch.stack([torch.ones_like(rad), 0.9 + 0.1 * r(n)], 1).float()
    weights = torch.exp(0.3 * torch.randn(n, device=dev, generator=g))
    weights[r(n) < 0.03] = 0.          # detectors cut for the whole observation
    return g, bore, dets, resp, weights


def _pix_shape(c):
    return (12 * c["nside"] ** 2,) if c["proj"] == "HP" else (c["ny"], c["nx"])


def _random_map(c, g, dev):
    return torch.randn((NCOMP[c["comps"]],) + _pix_shape(c), dtype=torch.float64, device=dev,
                       generator=g)


def _cut_mask(c, g, dev):
    """Samples kept: flags of about one glitch per 20000 samples (up to 200
    samples long) are cut."""
    n_det, n_time = c["n_det"], c["n_time"]
    n = max(1, n_det * n_time // 20000)
    edge = torch.zeros((n_det, n_time + 1), dtype=torch.int8, device=dev)
    d = torch.randint(n_det, (n,), device=dev, generator=g)
    a = torch.randint(n_time, (n,), device=dev, generator=g)
    b = torch.minimum(a + torch.randint(1, 200, (n,), device=dev, generator=g),
                      torch.tensor(n_time, device=dev))
    one = torch.ones(n, dtype=torch.int8, device=dev)
    edge.index_put_((d, a), one, accumulate=True)
    edge.index_put_((d, b), -one, accumulate=True)
    return torch.cumsum(edge[:, :-1], 1, dtype=torch.int8) <= 0


def _geom_args(c):
    if c["proj"] == "HP":
        return (c["nside"], c["nest"]) + ((c["tile"],) if c["tile"] else ())
    r = c["res"] * ARCMIN
    a = (c["ny"], c["nx"], r, -r, c["ny"] / 2. + 0.5, c["nx"] / 2. + 0.5)
    return a + ((c["tile"], c["tile"]) if c["tile"] else ())


def _engine(c):
    name = "ProjEng_%s_%s_%s%s" % (c["proj"], c["comps"], "Tiled" if c["tile"] else "NonTiled",
                                   "_Bilinear" if c["bilinear"] else "")
    eng = getattr(so3g, name)(_geom_args(c))
    if c["mode"] == "mixed":
        eng.pointing = _abi.POINTING_MIXED
    return eng


def _tile_slices(c):
    """Pixel slices of the tiles, in tile order."""
    if c["proj"] == "HP":
        n = 12 * c["tile"] ** 2
        k = 12 * c["nside"] ** 2 // n
        return [(slice(i * k, (i + 1) * k),) for i in range(n)]
    t = c["tile"]
    return [(slice(y, min(y + t, c["ny"])), slice(x, min(x + t, c["nx"])))
            for y in range(0, c["ny"], t) for x in range(0, c["nx"], t)]


def _tiles_of(c, lead, dev, whole=None):
    """(buffer, tiles): every tile a view of one flat buffer, from the whole
    map's values when given."""
    sizes = [tuple(s.stop - s.start for s in sl) for sl in _tile_slices(c)]
    n = math.prod(lead)
    buf = torch.zeros(n * sum(math.prod(s) for s in sizes), dtype=torch.float64, device=dev)
    tiles, at = [], 0
    for s in sizes:
        k = n * math.prod(s)
        tiles.append(buf[at:at + k].view(lead + s))
        at += k
    if whole is not None:
        for t, sl in zip(tiles, _tile_slices(c)):
            t.copy_(whole[(slice(None),) * len(lead) + sl])
    return buf, tiles


def _inputs(c, seed, dev):
    """Everything drawn from the seed, in one order."""
    g, bore, dets, resp, weights = _observation(c, seed, dev)
    q = _qmul(_native_rotation(c, dev), bore)
    d = dict(bore=bore, q=q.contiguous(), dets=dets.contiguous(), resp=resp,
             weights=weights if c["det_weights"] else None)
    if c["op"] in ("from_map", "grad"):
        d["map"] = _random_map(c, g, dev)
    if c["op"] in ("step", "to_map", "grad", "precomp"):
        d["signal"] = torch.randn((c["n_det"], c["n_time"]), device=dev, generator=g)
    d["mask"] = _cut_mask(c, g, dev) if c["cuts"] else None
    return d


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda", torch.cuda.current_device())
    s = _inputs(c, seed, dev)
    nc = NCOMP[c["comps"]]
    lead = (nc, nc) if c["op"] == "weights" else (nc,)
    st = dict(case=c, q=s["q"], dets=s["dets"], resp=s["resp"], weights=s["weights"],
              signal=s.get("signal"), map=s.get("map"), cuts=None)
    if c["op"] == "precomp":
        st["eng"] = so3g.ProjEng_Precomp_NonTiled()
        pix, spin = [], []
        for d0, d1, p, pf in _pointing(c, s, dev):
            pix.append(p.to(torch.int32))
            spin.append(pf.float())
        st["pix"], st["spin"] = torch.cat(pix), torch.cat(spin)
        return st
    if c["host"]:
        wcs = SimpleWCS(c["proj"], (-AZ0, c["el"]), (-c["res"] / 60, c["res"] / 60),
                        (c["nx"] / 2. + 0.5, c["ny"] / 2. + 0.5))
        p = Projectionist.for_geom((c["ny"], c["nx"]), wcs,
                                   interpol="bilinear" if c["bilinear"] else None)
        fp = proj_coords.FocalPlane(quats=s["dets"].cpu().numpy(), resps=s["resp"].cpu().numpy())
        asm = proj_coords.Assembly.attach(proj_quat.G3VectorQuat(s["bore"].cpu().numpy()), fp)
        st.update(projectionist=p, assembly=asm, signal=s["signal"].cpu().numpy(),
                  scanned=np.empty((c["n_det"], c["n_time"]), np.float32))
        return st
    st["eng"] = _engine(c)
    if s["mask"] is not None:
        st["cuts"] = RangesMatrix.from_mask(s["mask"])
    if c["tile"]:
        st["buffer"], st["tiles"] = _tiles_of(c, lead, dev, st["map"])
    if c["op"] == "grad":
        st["map"] = st["map"].requires_grad_(True)
    return st


def run(st):
    c = st["case"]
    if c["host"]:
        p, asm = st["projectionist"], st["assembly"]
        m = p.to_map(st["signal"], asm, comps=c["comps"])
        st["scanned"].fill(0.)
        p.from_map(m, asm, signal=st["scanned"], comps=c["comps"])
        return [m, st["scanned"]]
    eng = st["eng"]
    if c["op"] == "precomp":
        m = torch.zeros((NCOMP[c["comps"]],) + _pix_shape(c), dtype=torch.float64,
                        device=st["pix"].device)
        eng.to_map(m, st["pix"], st["spin"], st["signal"], None, None)
        return [m, eng.from_map(m, st["pix"], st["spin"], None)]
    point = (st["q"], st["dets"], st["resp"])
    if c["op"] == "grad":
        st["map"].grad = None
        s = autograd.from_map(eng, st["map"], *point)
        s.backward(st["signal"])
        return [s.detach(), st["map"].grad]
    if c["op"] == "from_map":
        return eng.from_map(st["tiles"] if c["tile"] else st["map"], *point, None)
    target = None
    if c["tile"]:
        target = st["tiles"]
        st["buffer"].zero_()
    if c["op"] == "weights":
        m = eng.to_weight_map(target, *point, st["weights"], st["cuts"])
    else:
        m = eng.to_map(target, *point, st["signal"], st["weights"], st["cuts"])
    out = st["buffer"] if c["tile"] else m
    if c["op"] == "step":
        return [out, eng.from_map(m, *point, None)]
    return out


def work(case):
    """Bytes: the signal and pointing read once, the signal written once, a
    map written (and read back) once.  Operations: per sample about 30 for a
    pixel and its spin factors from a smooth scan, and two per component and
    direction."""
    c = case
    n, nc = c["n_det"] * c["n_time"], NCOMP[c["comps"]]
    npix = math.prod(_pix_shape(c))
    point = 32 * c["n_time"] + 40 * c["n_det"]
    if c["op"] == "precomp":
        return {"bytes": (8 + 4 * nc) * n + 8 * n + 8 * nc * npix, "flops": 4 * nc * n}
    into = {"bytes": 4 * n + point + 8 * nc * npix, "flops": (30 + 2 * nc) * n}
    out = {"bytes": 4 * n + point + 8 * nc * npix, "flops": (30 + 2 * nc) * n}
    if c["op"] == "weights":
        return {"bytes": point + 8 * nc * nc * npix, "flops": (30 + nc * (nc + 1)) * n}
    if c["op"] == "to_map":
        return into
    if c["op"] == "from_map":
        return out
    # step, grad: both directions, the pointing read and evaluated once.
    return {"bytes": 8 * n + point + 8 * nc * npix * (2 if c["op"] == "grad" else 1),
            "flops": (30 + 4 * nc) * n}


# ---------------------------------------------------------------------------
# The same results in float64, without the library.

_LUT_N = 1 << 14     # knots of the asin and atan2 tables the projections are defined with


def _lut(table, x):
    d = x * (_LUT_N - 1)
    i = d.long().clamp_(0, _LUT_N - 2)
    f = d - i
    return table[i] * (1 - f) + table[i + 1] * f


def _lon_lat(q, tables):
    a, b, c, d = q.unbind(-1)
    z = a * a - b * b - c * c + d * d
    y, x = c * d - a * b, c * a + d * b
    ay, ax = y.abs(), x.abs()
    steep = ax < ay
    th = _lut(tables[1], torch.where(steep, ax, ay) / torch.where(steep, ay, ax))
    th = torch.where(steep, math.pi / 2 - th, th)
    th = torch.where(x < 0, math.pi - th, th)
    lat = torch.sign(z) * _lut(tables[0], z.abs())
    h2 = (1 - z * z) / 4
    nc, ns = a * c - b * d, c * d + a * b
    return torch.where(y < 0, -th, th), lat, (nc * nc - ns * ns) / h2, 2 * nc * ns / h2


def _planar(proj, q):
    a, b, c, d = q.unbind(-1)
    n = a * a + d * d
    u, v = a * b - c * d, a * c + b * d
    den = 2 * n - 1 if proj == "TAN" else torch.sqrt(n)
    co, si = (a * a - d * d) / n, 2 * a * d / n
    return 2 * u / den, 2 * v / den, co * co - si * si, 2 * co * si


def _spread(v):
    r = v & 0xffff
    for k, m in ((8, 0x00ff00ff), (4, 0x0f0f0f0f), (2, 0x33333333), (1, 0x55555555)):
        r = (r ^ (r << k)) & m
    return r


def _ang2pix(nside, nest, lon, lat):
    """HEALPix pixel of (lon, lat): the published ang2ring / ang2nest."""
    z, s = torch.sin(lat), torch.cos(lat)
    za = z.abs()
    x = lon / (2 * math.pi)
    tt = 4 * torch.where(x < 0, x + 1, x)
    jp, jm = 0.5 + tt - 0.75 * z, 0.5 + tt + 0.75 * z
    fp, fm = jp.long(), jm.long()
    fe = torch.where(fp == fm, fp | 4, torch.where(fp < fm, fp, fm + 8))
    nt = tt.long().clamp(max=3)
    tp, tmp = tt - nt, s / torch.sqrt((1 + za) / 3)
    cp, cm = (tp * tmp).clamp(max=1), ((1 - tp) * tmp).clamp(max=1)
    belt, north = za <= 2. / 3., z >= 0
    hx = torch.where(belt, jm - fm, torch.where(north, 1 - cm, cp))
    hy = torch.where(belt, 1 + fp - jp, torch.where(north, 1 - cp, cm))
    f = torch.where(belt, fe, torch.where(north, nt, nt + 8))
    ix, iy = (hx * nside).long(), (hy * nside).long()
    if nest:
        return f * nside * nside + _spread(ix) + 2 * _spread(iy)
    row = f // 4
    jr = (row + 2) * nside - ix - iy - 1
    jpll = 2 * (f % 4) + torch.where(row == 1, 0, 1)
    cap_n, cap_s = jr < nside, jr > 3 * nside
    rr = torch.where(cap_s, 4 * nside - jr, jr)
    nr = torch.where(cap_n | cap_s, rr, nside)
    odd = torch.where(cap_n | cap_s, 0, (jr - nside) & 1)
    j = torch.div(jpll * nr + ix - iy + 1 + odd, 2, rounding_mode="trunc")
    j = torch.where(j > 4 * nside, j - 4 * nside, torch.where(j < 1, j + 4 * nside, j))
    base = torch.where(cap_n, 2 * rr * (rr - 1),
                       torch.where(cap_s, 12 * nside * nside - 2 * (rr + 1) * rr,
                                   2 * nside * (nside - 1) + (jr - nside) * 4 * nside))
    return base + j - 1


def _chunks(c):
    rows = max(1, 20_000_000 // c["n_time"])
    return [(d, min(c["n_det"], d + rows)) for d in range(0, c["n_det"], rows)]


def _tables(dev):
    k = torch.arange(_LUT_N, dtype=torch.float64, device=dev) / (_LUT_N - 1)
    return torch.asin(k), torch.atan(k)


def _coords(c, s, d0, d1, tables):
    """Pixel coordinates (HP: pixel and None) and spin factors of detectors
    d0 to d1."""
    q = _qmul(s["q"][None], s["dets"][d0:d1, None])
    if c["proj"] in ("CAR", "HP"):
        X, Y, f1, f2 = _lon_lat(q, tables)
    else:
        X, Y, f1, f2 = _planar(c["proj"], q)
    r = s["resp"][d0:d1].double()
    T, P = r[:, :1].expand_as(f1), r[:, 1:]
    pf = {"T": [T], "QU": [P * f1, P * f2], "TQU": [T, P * f1, P * f2]}[c["comps"]]
    if c["proj"] == "HP":
        return _ang2pix(c["nside"], c["nest"], X, Y), None, pf
    res = c["res"] * ARCMIN
    return X / -res + c["nx"] / 2., Y / res + c["ny"] / 2., pf


def _taps(c, x, y):
    """(pixel index, weight or None, on the map) of each interpolation tap."""
    if y is None:
        return [(x, None, torch.ones_like(x, dtype=torch.bool))]
    ny, nx = c["ny"], c["nx"]
    x0, y0 = torch.floor(x), torch.floor(y)
    if c["tile"]:      # the tiled pixelizors truncate toward zero
        x0, y0 = torch.trunc(x), torch.trunc(y)
    if not c["bilinear"]:
        low = -1 if c["tile"] else 0
        on = (x > low) & (y > low) if c["tile"] else (x >= low) & (y >= low)
        on = on & (x < nx) & (y < ny)
        return [(torch.where(on, y0 * nx + x0, 0.).long(), None, on)]
    out = []
    for dy in (0, 1):
        for dx in (0, 1):
            # The weight x - x0 goes with x0 and 1 - (x - x0) with x0 + 1.
            w = (1 - (y - y0) if dy else y - y0) * (1 - (x - x0) if dx else x - x0)
            xx, yy = x0 + dx, y0 + dy
            on = (xx >= 0) & (xx < nx) & (yy >= 0) & (yy < ny)
            out.append((torch.where(on, yy * nx + xx, 0.).long(), w, on))
    return out


def _pointing(c, s, dev):
    """(d0, d1, (iy, ix) pixels, spin factors) of the stored pointing."""
    tables = _tables(dev)
    for d0, d1 in _chunks(c):
        x, y, pf = _coords(c, s, d0, d1, tables)
        ok = (x >= 0) & (x < c["nx"]) & (y >= 0) & (y < c["ny"])
        p = torch.stack([torch.where(ok, torch.floor(v), -1.) for v in (y, x)], -1)
        yield d0, d1, p, torch.stack(pf, -1)


def exact(case, seed):
    c = dict(case)
    dev = torch.device("cuda", torch.cuda.current_device())
    s = _inputs(c, seed, dev)
    tables, nc, npix = _tables(dev), NCOMP[c["comps"]], math.prod(_pix_shape(c))
    sig = s.get("signal")
    keep = s["mask"]
    det_wt = s["weights"]

    def pointing(d0, d1):
        x, y, pf = _coords(c, s, d0, d1, tables)
        if c["op"] == "precomp":
            pf = [v.float().double() for v in pf]     # stored as float32
        return _taps(c, x, y), pf

    def project():
        planes = nc * nc if c["op"] == "weights" else nc
        m = torch.zeros((planes, npix), dtype=torch.float64, device=dev)
        for d0, d1 in _chunks(c):
            taps, pf = pointing(d0, d1)
            for idx, w, on in taps:
                use = on if keep is None else on & keep[d0:d1]
                v = use.double() if sig is None else sig[d0:d1].double() * use
                if w is not None:
                    v = v * w
                if det_wt is not None:
                    v = v * det_wt[d0:d1, None].double()
                idx = idx.reshape(-1)
                if c["op"] == "weights":
                    if w is not None:
                        v = v * w
                    for i in range(nc):
                        for j in range(i, nc):
                            m[i * nc + j].index_add_(0, idx, (v * pf[i] * pf[j]).reshape(-1))
                else:
                    for i in range(nc):
                        m[i].index_add_(0, idx, (v * pf[i]).reshape(-1))
        lead = (nc, nc) if c["op"] == "weights" else (nc,)
        return m.view(lead + _pix_shape(c))

    def scan(m):
        m = m.view(nc, npix)
        out = torch.empty((c["n_det"], c["n_time"]), dtype=torch.float64, device=dev)
        for d0, d1 in _chunks(c):
            taps, pf = pointing(d0, d1)
            o = torch.zeros_like(pf[0])
            for idx, w, on in taps:
                v = sum(m[i][idx] * pf[i] for i in range(nc))
                o += torch.where(on, v if w is None else v * w, 0.)
            out[d0:d1] = o
        return out

    def laid(m):
        """A map as run() gives it."""
        if not c["tile"]:
            return m
        lead = (nc, nc) if c["op"] == "weights" else (nc,)
        return _tiles_of(c, lead, dev, m)[0]

    if c["op"] == "from_map":
        return scan(s["map"])
    m = project()
    if c["op"] in ("to_map", "weights"):
        return laid(m)
    if c["op"] == "grad":
        return [scan(s["map"]), m]
    return [laid(m), scan(m)]
