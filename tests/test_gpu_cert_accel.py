"""Chunked certified pointing of scans that accelerate: the second-order terms
of a chunk are not small against the square of the first-order ones, at the
vertex of a parabola least of all.  from_map bit for bit the general
kernels', to_map up to the order of the float64 additions (1e-12 of the map's
scale)."""
import numpy as np
import pytest

import so3g_gb300 as so3g
from so3g_gb300.proj import quat
from conftest import bits_equal
from test_gpu_cert_chunked import _both

pytestmark = pytest.mark.gpu

DEG = np.pi / 180
N_DET, N_TIME = 200, 20_037


def _path(geom, acc, noise):
    """Parabolas of `acc` deg/s^2, 389 samples each, along a slanted line."""
    rng = np.random.default_rng(5)
    t = (np.arange(N_TIME) % 389 - 194.3) / 200.
    s = 0.5 * acc * t * t
    if geom in ("CAR", "HP"):
        q = np.asarray(quat.rotation_lonlat((3 + .8 * s) * DEG, (25 + .6 * s) * DEG, .3 + 0 * s))
    else:
        q = np.asarray(quat.rotation_xieta((2 + .8 * s) * DEG, (3 - .6 * s) * DEG, .3 + 0 * s))
    if noise:
        q = q + noise * rng.standard_normal(q.shape)
        q /= np.sqrt((q * q).sum(1, keepdims=True))
    return q


@pytest.mark.parametrize("noise", [0., 1e-9, 2e-8])
@pytest.mark.parametrize("acc", [.3, 1., 4.])
@pytest.mark.parametrize("geom", ["CAR", "HP", "TAN", "ZEA", "SIN"])
def test_vertices(gpulib, geom, acc, noise):
    import torch
    k = np.arange(N_DET)
    r, a = 3. * DEG * np.sqrt((k + .5) / N_DET), 2.4 * k
    dets = np.asarray(quat.rotation_xieta(r * np.cos(a), r * np.sin(a), 0.7 * k))
    resp = np.stack([np.ones(N_DET), 1 - 0.001 * k], 1).astype(np.float32)
    args = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
            for x in (_path(geom, acc, noise), dets, resp)]
    if geom == "HP":
        eng, shape = so3g.ProjEng_HP_QU_NonTiled((2048, True)), (12 << 22,)
    else:
        shape = (1200, 1300)
        at = (600.5 - 60 * 25, 650.5) if geom == "CAR" else (600.5, 650.5)
        eng = getattr(so3g, "ProjEng_%s_QU_NonTiled" % geom)(
            shape + (DEG / 60, -DEG / 60) + at)
    g = torch.Generator(device="cuda").manual_seed(1)
    m = torch.randn((2,) + shape, dtype=torch.float64, device="cuda", generator=g)
    sig = torch.zeros((N_DET, N_TIME), dtype=torch.float32, device="cuda")
    chunked, general = _both(lambda: eng.from_map(m, *args, sig.clone()))
    assert float((general != 0).float().mean()) > 0.5
    assert bits_equal(chunked.cpu().numpy(), general.cpu().numpy())
    ones = torch.ones_like(sig)
    a, b = _both(lambda: eng.to_map(torch.zeros_like(m), *args, ones))
    assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())
