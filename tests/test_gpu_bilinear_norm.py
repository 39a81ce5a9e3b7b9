"""Chunked bilinear from_map of boresights whose residual from the chunk
model has a part that is no rotation: stored in 32 bits, noise that is not
renormalised, an accelerating scan with jittering time stamps.  That part
scales the projection plane's coordinates, so it moves pixels far from the
map's centre.

On a checkerboard of +1 and -1 a sample is the alternating sum of its four
weights.  The chunked kernels' coordinates are within 2.5e-7 pixel of the
exact ones and the general kernels' within 1e-7: the sums differ by at most
2 (dx + dy) = 1.4e-6, by the weights' float32 products (3 roundings of at
most 2^-25 each, 4 weights, both kernels) and by the sums' (4 additions of
at most 2^-24, both kernels)."""
import numpy as np
import pytest

import so3g_gb300 as so3g
from so3g_gb300 import _abi, synth
from so3g_gb300.proj import quat
from conftest import bits_equal
from test_gpu_cert_chunked import _both

pytestmark = pytest.mark.gpu

DEG = np.pi / 180
N_DET, N_TIME = 24, 8000
TOL = 1.4e-6 + 2 * (12 * 2.0**-25 + 4 * 2.0**-24)


def _scan(boresight):
    """+-5 deg in longitude about a path 3 deg off the map's centre."""
    rng = np.random.default_rng(3)
    t = np.arange(N_TIME) / 200.
    if boresight == "accelerating":
        t = (1.7e9 + t) - 1.7e9      # spaced by 2.4e-7 s
        x = -4.5 + 0.02 * t + 0.5 * 0.01 * t * t
    else:
        s = (t + 0.7) % 20.
        x = np.where(s < 10., s, 20. - s) - 5.
    # (The native pole, the map's centre, is the focal plane's direction at 0.)
    q = np.asarray(quat.rotation_xieta(x * DEG, 3. * DEG + 0. * x, 0.2 + 0. * x))
    if boresight == "float32":
        q = q.astype(np.float32).astype(float)
    elif boresight in ("noise", "unit-noise"):
        q = q + (1e-8 if boresight == "noise" else 2e-8) * rng.standard_normal(q.shape)
        if boresight == "unit-noise":
            q /= np.sqrt((q * q).sum(1, keepdims=True))
    return q


def _call(proj, boresight, norm=1., res=.5):
    """(engine, map, arguments): a checkerboard of `res` arcmin pixels."""
    import torch
    k = np.arange(N_DET)
    r, a = 1. * DEG * np.sqrt((k + .5) / N_DET), 2.4 * k
    dets = np.asarray(quat.rotation_xieta(r * np.cos(a), r * np.sin(a), 0.7 * k))
    dets = dets * np.sqrt(norm)
    resp = np.ones((N_DET, 2), np.float32)
    args = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (_scan(boresight), dets, resp)]
    ny, nx = (1201, 1502) if res >= .5 else (2001, 2502)
    eng = getattr(so3g, "ProjEng_%s_T_NonTiled_Bilinear" % proj)(
        (ny, nx, res * synth.ARCMIN, -res * synth.ARCMIN, ny / 2. + .5, nx / 2. + .5))
    yx = torch.arange(ny, device="cuda")[:, None] + torch.arange(nx, device="cuda")
    return eng, (1. - 2. * (yx % 2)).double()[None].contiguous(), args


@pytest.mark.parametrize("boresight", ["unit", "float32", "noise", "accelerating"])
@pytest.mark.parametrize("proj", ["TAN", "ZEA", "SIN"])
def test_residual_norm(gpulib, proj, boresight):
    _check_mixed(*_call(proj, boresight))


@pytest.mark.parametrize("norm", [1.00098, 0.99905])
@pytest.mark.parametrize("proj", ["TAN", "ZEA", "SIN"])
def test_detector_norm(gpulib, proj, norm):
    """The residual's turn, with detector quaternions off unit length."""
    _check_mixed(*_call(proj, "unit-noise", norm))


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("proj", ["TAN", "ZEA", "SIN"])
def test_short_last_chunk(gpulib, proj, seed):
    """A last chunk of one sample, its model's other samples the chunk before's,
    with pointing noise: a polynomial through the one sample it is used at,
    with noise in every order."""
    import torch
    n = 64 * 200 + 1
    s = np.abs((np.arange(n) - n + 700) / 200. * 1.4 % 18. - 9.) - 4.5
    q = np.asarray(quat.rotation_xieta(s * DEG, 1. * DEG + 0. * s, 0.2 + 0. * s))
    q[-65:] += 3e-8 * np.random.default_rng(seed).standard_normal((65, 4))
    q /= np.sqrt((q * q).sum(1, keepdims=True))
    eng, m, args = _call(proj, "unit", res=.3)
    args[0] = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    _check_mixed(eng, m, args)


def _check_mixed(eng, m, args):
    eng.pointing = _abi.POINTING_MIXED
    chunked, general = _both(lambda: eng.from_map(m, *args, None))
    assert float((general != 0).float().mean()) > 0.3
    assert float((chunked.double() - general.double()).abs().max()) <= TOL


@pytest.mark.parametrize("proj", ["TAN", "ZEA", "SIN"])
def test_default_mode_weights(gpulib, proj):
    """In the default mode a weight is the float32 nearest the double-float
    coordinates' weight at every call size."""
    eng, m, args = _call(proj, "unit")
    chunked, general = _both(lambda: eng.from_map(m, *args, None))
    assert float((general != 0).float().mean()) > 0.3
    assert bits_equal(chunked.cpu().numpy(), general.cpu().numpy())
