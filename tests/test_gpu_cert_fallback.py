"""Calls whose samples the chunk models would leave to the per-sample path:
boresights or detectors stored in 32 bits, pointing noise, interpolation
between knots, scans over a pole.  They take the general kernels: the same
results, and about their time (they took 2 to 3 times it when every such
sample went through the chunked kernels' fallback; the limit lies between)."""
import numpy as np
import pytest

import so3g_gb300 as so3g
from so3g_gb300 import _abi, synth
from so3g_gb300.proj import quat
from conftest import bits_equal
from test_gpu_cert_chunked import _both

pytestmark = pytest.mark.gpu

DEG = np.pi / 180
N_DET, N_TIME = 64, 200_000
CASES = [("CAR", "TQU", "float32"), ("HP", "TQU", "float32"), ("CAR", "T", "noise3e-7"),
         ("HP", "T", "noise3e-7"), ("HP", "TQU", "knots200"), ("HP", "T", "knots200"),
         ("CAR", "TQU", "pole"), ("ZEA", "QU", "noise3e-7"), ("ZEA-bilinear", "TQU", "float32")]


def _call(geom, comps, boresight):
    import torch
    rng = np.random.default_rng(11)
    dets, _, _ = synth.focal_plane(rng, N_DET, 1.5)
    resp = np.stack([np.ones(N_DET), rng.uniform(.9, 1., N_DET)], 1).astype(np.float32)
    t = np.arange(N_TIME) / 200.
    s = t % 20.
    s = np.where(s < 10., s, 20. - s) - 5.
    lat = 85. if boresight == "pole" else 30.
    if geom.startswith("ZEA"):
        q = np.asarray(quat.rotation_xieta(s * DEG, (3. + 0. * s) * DEG, 0.2 + 0. * s))
    else:
        q = np.asarray(quat.rotation_lonlat(s / np.cos(lat * DEG) * DEG, (lat + .2 * s) * DEG,
                                            0.3 + 0. * s))
    if boresight == "float32":
        q = q.astype(np.float32).astype(float)
    elif boresight.startswith("noise"):
        q = q + float(boresight[5:]) * rng.standard_normal(q.shape)
        q /= np.sqrt((q * q).sum(1, keepdims=True))
    elif boresight.startswith("knots"):
        k = np.append(np.arange(0, N_TIME, 200), N_TIME - 1)
        q = np.stack([np.interp(np.arange(N_TIME), k, q[k, c]) for c in range(4)], 1)
    res = DEG / 60
    if geom == "HP":
        eng, shape = getattr(so3g, "ProjEng_HP_%s_NonTiled" % comps)((1024, False)), (12 << 20,)
    else:
        kind, _, bil = geom.partition("-")
        shape = (1500, 2000)
        at = 750.5 - 60 * (lat if kind == "CAR" else 0.)
        eng = getattr(so3g, "ProjEng_%s_%s_NonTiled%s" % (kind, comps, "_Bilinear" if bil else ""))(
            shape + (res, -res, at, 1000.5))
        if bil:
            eng.pointing = _abi.POINTING_MIXED
    m = torch.randn((eng.comp_count,) + shape, dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(2))
    return eng, m, [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (q, dets, resp)]


def _time(call):
    import torch
    out = []
    for _ in range(9):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        call()
        b.record()
        torch.cuda.synchronize()
        out.append(a.elapsed_time(b))
    return min(out[2:])     # (the host may stall in some)


@pytest.mark.parametrize("geom,comps,boresight", CASES)
def test_fallback(gpulib, geom, comps, boresight):
    import torch
    eng, m, args = _call(geom, comps, boresight)
    sig = torch.zeros((N_DET, N_TIME), dtype=torch.float32, device="cuda")
    chunked, general = _both(lambda: eng.from_map(m, *args, sig.clone()))
    assert float((general != 0).float().mean()) > 0.2
    assert bits_equal(chunked.cpu().numpy(), general.cpu().numpy())
    calls = [lambda: eng.from_map(m, *args, sig)]
    if geom != "ZEA-bilinear":
        dest = torch.zeros_like(m)
        calls.append(lambda: eng.to_map(dest, *args, sig))
    for call in calls:
        now, before = _both(lambda: _time(call))
        assert now < 1.5 * before
