"""Calls after, beside and between calls that raise: the error records kept
per thread for the next call are clean ones, on any stream and thread."""
import threading

import numpy as np
import pytest

import so3g_gb300 as so3g
from so3g_gb300.proj import quat

pytestmark = pytest.mark.gpu

DEG = np.pi / 180
NY, NX, TILE = 64, 96, 32


class _Tiled:
    """A tiled map whose second tile's samples are asked for or not."""

    def __init__(self):
        import torch
        t = np.arange(2000) / 2000.
        q = np.asarray(quat.rotation_lonlat((t * 4 - 2) * DEG, (t - .5) * DEG, 0. * t))
        dets = np.asarray(quat.rotation_xieta(np.array([0., .001]), np.array([0., .001])))
        self.args = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (
            q, dets, np.ones((2, 2), np.float32))]
        res = .1 * DEG
        self.eng = so3g.ProjEng_CAR_T_Tiled((NY, NX, res, -res, NY / 2. + .5, NX / 2. + .5,
                                             TILE, TILE))
        self.sig = torch.ones((2, 2000), dtype=torch.float32, device="cuda")

    def tiles(self, missing):
        import torch
        n = (NY // TILE) * (NX // TILE)
        hole = 1     # on the path
        return [None if missing and i == hole else
                torch.zeros((1, TILE, TILE), dtype=torch.float64, device="cuda")
                for i in range(n)]

    def clean(self):
        m = self.eng.to_map(self.tiles(False), *self.args, self.sig)
        return float(sum(t.sum() for t in m))

    def broken(self):
        with pytest.raises(RuntimeError, match="non-instantiated tile"):
            self.eng.to_map(self.tiles(True), *self.args, self.sig)


def test_call_after_an_error(gpulib):
    c = _Tiled()
    hits = c.clean()
    assert hits > 1000
    for _ in range(10):
        c.broken()
        assert c.clean() == hits
        assert c.clean() == hits


def test_two_streams(gpulib):
    import torch
    c = _Tiled()
    hits = c.clean()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for k in range(10):
        with torch.cuda.stream(streams[k % 2]):
            c.broken()
        with torch.cuda.stream(streams[(k + 1) % 2]):
            assert c.clean() == hits
        with torch.cuda.stream(streams[k % 2]):
            assert c.clean() == hits


def test_two_threads(gpulib):
    import torch
    c = _Tiled()
    hits = c.clean()
    torch.cuda.synchronize()
    wrong = []

    def work(kind):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for k in range(30):
                    if kind == "broken" or (kind == "both" and k % 2):
                        c.broken()
                    elif c.clean() != hits:
                        wrong.append(kind)
        except BaseException as e:      # noqa: B902 (pytest.raises' failure too)
            wrong.append("%s: %r" % (kind, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in ("clean", "broken", "both")]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
