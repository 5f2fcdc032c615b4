"""The short-range wake's kernels at the edges of their sizes: bunches that end
inside a warp, a tile or a chunk, more and fewer bins than a CTA's threads, the
extremes of z at lost particles (particle 0 among them); bins and kicks against
the oracle, a turn against its staged calls.  Tolerance of the kick: 1e-12 of
the largest (200 terms of a sum, 2^-53 each)."""
import ctypes as C

import numpy as np
import pytest

from cetasim_b200 import _abi
from helpers import pair, particles, small

pytestmark = pytest.mark.gpu


def _case(sizes, bins, **over):
    wl = small("large_trapping", 0.01, flag_beam_ion=0, flag_lr_wake=0, flag_fir=0, sr_bins=bins, **over)
    m = len(sizes)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:m].copy(), wl.harm[:m].copy(), wl.ne[:m].copy()
    wl.n_macro[:] = sizes
    parts = particles(wl, seed=23)
    surv = [np.zeros(n, dtype=np.uint8) for n in sizes]
    for j, (c, s) in enumerate(zip(parts, surv)):
        if len(s) > 4:
            s[1::5] = 1
            c[4, 1::5] *= 3.0  # lost ones beyond the survivors' range
        if j % 2 and len(s) > 4:
            s[0] = 1  # the range is seeded with particle 0, lost or not
            c[4, 0] = 8 * np.std(c[4])
    return wl, parts, surv


@pytest.mark.parametrize("bins", [7, 100, 300])
def test_bins_and_kick(bins):
    sizes = [2, 31, 257, 2049, 9001]
    wl, parts, surv = _case(sizes, bins)
    g, o = pair(wl, parts, surv)
    for turn in range(2):  # the potentials build on those of the turn before
        for b in (g, o):
            b.MPBeamRMSCal(0)
            before = [b.download(j)[0] for j in range(len(sizes))]
            b.SRWakeBeamIntaction(turn)
        for j, n in enumerate(sizes):
            have, want = g.download(j)[0], o.download(j)[0]
            kick = np.max(np.abs(want[5] - before[j][5]))
            assert np.array_equal(have[:5], want[:5])
            assert np.max(np.abs(have[5] - want[5])) <= 1e-12 * kick + 2.0**-53 * np.max(np.abs(want[5]))
            z, dz, cnt = C.c_double(), C.c_double(), np.zeros(bins, dtype=np.int32)
            g._check(g.lib.cg_sr_bins(g.h, j, C.byref(z), C.byref(dz), _abi.ptr(cnt)))
            idx = np.trunc((parts[j][4] - z.value) / dz.value).astype(int)
            idx = idx[(idx >= 0) & (idx < bins)]
            assert np.array_equal(cnt, np.bincount(idx, minlength=bins))


@pytest.mark.parametrize("xy", [False, True])
def test_turn_repeats_the_staged_calls(xy):
    wl, parts, surv = _case([33, 257, 2049, 5000], 100)
    beams = []
    for staged in (False, True):
        b = pair(wl, parts, surv)[0]
        if xy:
            b.lib.cg_set_sr_potentials(b.h, 1)
        if staged:
            for k in range(wl.cfg.n_sections):
                b.BeamTransferPerInteractionPointDueToLatticeT(k)
            b.MPBeamRMSCal(wl.cfg.n_sections - 1)
            b.BeamMomtumUpdateDueToRFTest()
            b.BeamLongiPosTransferOneTurn()
            b.BeamEnergyLossOneTurn()
            b.BeamSynRadDamping(0)
            b.SRWakeBeamIntaction(0)
            b.MarkParticleLostInBunch()
        else:
            b.Run(0, 1)
        beams.append(b)
    for j in range(4):
        (ca, sa), (cb, sb) = beams[0].download(j), beams[1].download(j)
        assert np.array_equal(ca, cb) and np.array_equal(sa, sb)
