"""Chunked certified pointing of quaternions that are not of unit length.
The exact path takes sin(lat) = a^2 - b^2 - c^2 + d^2 of the quaternion as
it is, so its norm moves the latitude of CAR and HEALPix pixels: boresights
interpolated between knots and not renormalised, stored in 32 bits, or of a
constant norm off 1, and detector quaternions off 1.  Every term must be the
general certified kernels': from_map bit for bit, to_map and to_weight_map
up to the order of the float64 additions (1e-12 of the map's scale)."""
import numpy as np
import pytest

import so3g_gb300 as so3g
from so3g_gb300.proj import quat
from test_gpu_cert_chunked import _both

pytestmark = pytest.mark.gpu

DEG = np.pi / 180
N_DET, N_TIME = 40, 6000
BORESIGHTS = ["unit", "knots200", "knots1000", "norm1e-5", "norm4e-4", "float32", "dets1e-4"]


def _path(lat):
    """A 1 deg/s triangle scan of +-2 deg, at 45 degrees to the meridian."""
    s = (np.arange(N_TIME) / 200. + 0.3) % 8.
    s = np.where(s < 4., s, 8. - s) - 2.
    return np.asarray(quat.rotation_lonlat(s * np.sqrt(.5) / np.cos(lat * DEG) * DEG,
                                           (lat + s * np.sqrt(.5)) * DEG, 0.3 + 0 * s))


def _knots(q, step):
    t = np.arange(len(q), dtype=float)
    k = np.append(np.arange(0, len(q), step), len(q) - 1)
    return np.stack([np.interp(t, k, q[k, c]) for c in range(4)], 1)


def _pointing(lat, boresight):
    q = _path(lat)
    k = np.arange(N_DET)
    r, a = 1.5 * DEG * np.sqrt((k + .5) / N_DET), 2.4 * k
    dets = np.asarray(quat.rotation_xieta(r * np.cos(a), r * np.sin(a), 0.7 * k))
    if boresight.startswith("knots"):
        q = _knots(q, int(boresight[5:]))
    elif boresight.startswith("norm"):
        q = q * np.sqrt(1 + float(boresight[4:]))
    elif boresight == "float32":
        q = q.astype(np.float32).astype(float)
    elif boresight.startswith("dets"):
        dets = dets * np.sqrt(1 + float(boresight[4:]))
    resp = np.stack([np.ones(N_DET), 1 - 0.01 * k], 1).astype(np.float32)
    return q, dets, resp


def _engine(geom, comps, lat):
    kind, _, tiled = geom.partition("-")
    if kind == "HP":
        return getattr(so3g, "ProjEng_HP_%s_NonTiled" % comps)((2048, tiled == "NEST"))
    # 1 arcmin pixels around (lat, 0); native (0, 0) is off the map.
    wcs = (600, 601, DEG / 60, -DEG / 60, 300.5 - 60 * lat, 301.)
    return getattr(so3g, "ProjEng_CAR_%s_%s" % (comps, "Tiled" if tiled else "NonTiled"))(
        wcs + ((100, 90) if tiled else ()))


def _bits(pair):
    import torch
    return torch.equal(pair[0].view(torch.int32), pair[1].view(torch.int32))


def _close(pair):
    a, b = (m if isinstance(m, list) else [m] for m in pair)
    top = max(float(t.abs().max()) for t in b)
    return top > 0 and max(float((x - y).abs().max()) for x, y in zip(a, b)) <= 1e-12 * top


@pytest.mark.parametrize("lat", [20., 50., 75.])
@pytest.mark.parametrize("comps", ["T", "QU", "TQU"])
@pytest.mark.parametrize("geom", ["CAR", "CAR-tiled", "HP-RING", "HP-NEST"])
def test_norms(gpulib, geom, comps, lat):
    import torch
    g = torch.Generator(device="cuda").manual_seed(7)
    eng = _engine(geom, comps, lat)
    nc = eng.comp_count
    sizes = [(600, 601)]
    if geom == "CAR-tiled":
        sizes = [(min(100, 600 - y), min(90, 601 - x)) for y in range(0, 600, 100)
                 for x in range(0, 601, 90)]
    elif geom != "CAR":
        sizes = [(12 * 2048 ** 2,)]

    def new(*lead):
        m = [torch.zeros(lead + s, dtype=torch.float64, device="cuda") for s in sizes]
        return m if geom == "CAR-tiled" else m[0]

    m = new(nc)
    for t in (m if isinstance(m, list) else [m]):
        t.normal_(generator=g)
    sig = torch.randn((N_DET, N_TIME), device="cuda", generator=g)
    wrong = []
    for boresight in BORESIGHTS:
        args = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
                for x in _pointing(lat, boresight)]
        pair = _both(lambda: eng.from_map(m, *args, sig.clone()))
        assert float((pair[1] != sig).float().mean()) > 0.3
        if not _bits(pair):
            wrong.append("from_map " + boresight)
        if not _close(_both(lambda: eng.to_map(new(nc), *args, sig))):
            wrong.append("to_map " + boresight)
        if not geom.startswith("HP") and not _close(
                _both(lambda: eng.to_weight_map(new(nc, nc), *args))):
            wrong.append("to_weight_map " + boresight)
    assert not wrong
