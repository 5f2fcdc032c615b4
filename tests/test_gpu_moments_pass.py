"""Moments by pivoted sums (k_moments, the map pass, the caller-buffer call) at
the sizes where a warp, a step, a tile or a chunk ends, with the first
particles lost (the pivot comes later) and with a centroid far outside the
bunch.  Tolerance against 80-bit sums: 1e-13, some hundred roundings of the
2^-53 of a sum whose pivot lies within a sigma of the mean, and for the
centroid 60 sigma away the same relative to it."""
import ctypes as C

import numpy as np
import pytest

from cetasim_b200 import _abi
from cetasim_b200.beam import MPBeam
from helpers import particles, small

pytestmark = pytest.mark.gpu


def _want(c, s, beta):
    v = c[:, s == 0].astype(np.longdouble)
    m = v.mean(axis=1)
    d = v - m[:, None]
    out = {"mean": m, "n": v.shape[1]}
    e = []
    for i in (0, 2, 4):
        a, b, ab = (d[i] ** 2).mean(), (d[i + 1] ** 2).mean(), (d[i] * d[i + 1]).mean()
        e.append(np.sqrt(a * b - ab * ab))
    out["emit"], out["sz"], out["sdp"] = e, np.sqrt((d[4] ** 2).mean()), np.sqrt((d[5] ** 2).mean())
    z = np.append(c[4][s == 0], c[4, 0])
    out["z"] = z.min() - 1e-6, z.max() + 1e-6
    return out


def _check(m, w, n):
    assert m.n_alive == w["n"] and m.n_macro == n
    scale = [np.sqrt(w["emit"][0] * 10), np.sqrt(w["emit"][0] / 10), np.sqrt(w["emit"][1] * 10),
             np.sqrt(w["emit"][1] / 10), w["sz"], w["sdp"]]
    for i in range(6):
        assert abs(m.mean[i] - w["mean"][i]) <= 1e-13 * max(abs(w["mean"][i]), scale[i])
    for i in range(3):
        assert abs(m.emit[i] - w["emit"][i]) <= 1e-12 * w["emit"][i]
    assert abs(m.bunch_length - w["sz"]) <= 1e-13 * w["sz"]
    assert abs(m.energy_spread - w["sdp"]) <= 1e-13 * w["sdp"]
    assert m.z_min == w["z"][0] and m.z_max == w["z"][1]


@pytest.mark.parametrize("n,lost,off", [(33, 0, 0), (127, 5, 0), (128, 0, 0), (129, 128, -1), (256, 130, 0),
                                        (257, 31, 60), (2049, 300, 0), (5000, 1100, 60),
                                        (70001, 257, 0), (600000, 2000, 60)])
def test_moments(n, lost, off):
    wl = small("plain_single", n / 1e5)
    wl.n_macro[0] = n
    c = particles(wl, seed=n)[0]
    s = np.zeros(n, dtype=np.uint8)
    if off < 0:  # every particle but the last few lost
        c, s = np.concatenate([c, c[:, :0]], 1), s
        lost = n - 100
    s[:lost] = 1
    c[:, :lost] *= 1e3  # lost particles far away must not enter
    c += max(off, 0) * np.std(c[:, lost:], axis=1)[:, None]
    c[4, 0] = c[4, lost]  # the z range is seeded with particle 0, lost or not
    g = MPBeam(wl)
    g.upload(0, c, s)
    g.MPBeamRMSCal(0)
    want = _want(c, s, 10.0)
    _check(g.moments()[0], want, n)
    # the caller-buffer call
    if n <= 1048576:
        import torch
        d, f = torch.from_numpy(c).cuda(), torch.from_numpy(s).cuda()
        o = torch.zeros(C.sizeof(_abi.BunchMoments), dtype=torch.uint8, device="cuda")
        rc = _abi.load().cg_bunch_moments_noalloc(d.data_ptr(), n, f.data_ptr(), n, 10.0, 10.0,
                                                  o.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        _check(_abi.BunchMoments.from_buffer_copy(o.cpu().numpy().tobytes()), want, n)
    # the map pass leaves the moments that k_moments makes of its particles
    t = C.c_double()
    g._check(g.lib.cg_time_stage(g.h, 5, 0, 1, C.byref(t)))
    a = bytes(g.moments())
    g.MPBeamRMSCal(0)
    assert a == bytes(g.moments())


@pytest.mark.parametrize("n,lost", [(45, 0), (300, 7), (5000, 1100), (70001, 257)])
def test_equal_coordinates_have_zero_size(n, lost):
    """A coordinate that is the same in every alive particle: its mean is that
    value and its size zero exactly (a zero size is an error further on)."""
    wl = small("plain_single", n / 1e5)
    wl.n_macro[0] = n
    c = particles(wl, seed=n)[0]
    s = np.zeros(n, dtype=np.uint8)
    s[:lost] = 1
    c[4, lost:], c[5, lost:] = 1.1e-3, 0.7e-4
    g = MPBeam(wl)
    g.upload(0, c, s)
    g.MPBeamRMSCal(0)
    m = g.moments()[0]
    assert (m.bunch_length, m.energy_spread) == (0.0, 0.0)
    assert (m.mean[4], m.mean[5]) == (1.1e-3, 0.7e-4)
