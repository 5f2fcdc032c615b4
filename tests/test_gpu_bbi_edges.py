"""The broadband-impedance kernels at the edges of their sizes: bunches over
fewer and more bins than a CTA counts in shared memory, bunches that end
inside a warp, a tile or a chunk, profiles that reach the filter's ends, and
the loss check that ends the kick; one kick and its potentials against the
oracle, whole turns against their staged calls.  Tolerance: 1e-11 of the
largest kick or potential, as against the reference's runs."""
import numpy as np
import pytest

import bbicases
from cetasim_b200 import configs
from helpers import pair, particles

pytestmark = pytest.mark.gpu


def _train(sizes, stretch, td, rows, **over):
    wl = configs.make("fast_ion", n_scale=0.01)
    m = len(sizes)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:m].copy(), wl.harm[:m].copy(), wl.ne[:m].copy()
    wl.n_macro[:] = sizes
    c = wl.cfg
    c.flag_beam_ion = c.flag_lr_wake = c.flag_fir = c.flag_sr_wake = 0
    for k, v in over.items():
        setattr(c, k, v)
    r = c.ring
    bucket = r.t0 * 299792458.0 / r.harmonics
    if td:
        wl.set_bbi(bbicases.wake_table(rows, 0.9 * bucket / 2500, rows // 3), 1)
    else:
        # rows frequencies give bins of c / (2 fmax): the profile spans 1.2 buckets
        fmax = 299792458.0 * (rows - 1) / (1.2 * bucket)
        wl.set_bbi(bbicases.resonator_table(rows, fmax), 0)
    parts = particles(wl, seed=17)
    for p in parts:
        p[4] *= stretch
        np.clip(p[4], -0.49 * bucket, 0.49 * bucket, out=p[4])
    return wl, parts


CASES = [(0, 1.0, 1300), (0, 12.0, 1300), (0, 40.0, 1700), (1, 1.0, 300), (1, 16.0, 900), (1, 40.0, 900)]
SIZES = [1, 31, 257, 2049, 9000]


# the kicks of the longer bunches with a wake table are below a momentum's
# rounding over the tolerance: their potentials are compared
@pytest.mark.parametrize("td,stretch,rows", CASES[:4])
def test_kick(td, stretch, rows):
    wl, parts = _train(SIZES, stretch, td, rows)
    g, o = pair(wl, parts)
    for b in (g, o):
        b.BBImpBeamInteraction()
    for j, p in enumerate(parts):
        have, want = g.download(j)[0], o.download(j)[0]
        for q in range(6):
            k = np.max(np.abs(want[q] - p[q]))
            assert np.max(np.abs(have[q] - want[q])) <= 1e-11 * k


@pytest.mark.parametrize("td,stretch,rows", CASES)
def test_profile_and_potentials(td, stretch, rows):
    wl, parts = _train(SIZES, stretch, td, rows)
    g, o = pair(wl, parts)
    for b in (g, o):
        b.BBImpBeamInteraction()
    for j in range(len(parts)):
        a, have = g.bbi_profile(j)
        want = o.bbi_profile(j)[:, a:a + have.shape[1]]
        assert np.max(np.abs(have[0] - want[0])) <= 1e-11 * np.max(np.abs(want[0]))
        for q in range(1, 6):
            kept = have[q] != 0  # at most the bins between the first and the last particle's
            k = np.max(np.abs(want[q][kept]), initial=0.0)
            assert np.max(np.abs(have[q] - want[q])[kept], initial=0.0) <= 1e-11 * k


@pytest.mark.parametrize("lr", [0, 1])
def test_turn_repeats_the_staged_calls(lr):
    wl, parts = _train([33, 257, 2049], 1.0, 0, 900, flag_lr_wake=lr, lr_turns=4,
                       lr_bbr=configs.bbr([(0.0, 1.0, 1.2e9, 1e6, 1e4, 1.2e9, 1e6, 1e4, 1.2e9)]))
    z_loss = wl.cfg.ring.t0 * 299792458.0 / wl.cfg.ring.harmonics / 2
    for p in parts:
        p[4, ::9] += 0.9999 * z_loss  # some drift out of the bucket, none out of the profile
    a, _ = pair(wl, parts)
    b, _ = pair(wl, parts)
    a.Run(0, 1)
    for k in range(wl.cfg.n_sections):
        b.BeamTransferPerInteractionPointDueToLatticeT(k)
    if lr:
        b.MPBeamRMSCal(wl.cfg.n_sections - 1)
    b.BeamMomtumUpdateDueToRFTest()
    b.BeamLongiPosTransferOneTurn()
    b.BeamEnergyLossOneTurn()
    b.BeamSynRadDamping(0)
    b.BBImpBeamInteraction()
    if lr:
        b.LRWakeBeamIntaction()
    t = np.asarray(b.MarkParticleLostInBunch())
    for j in range(wl.n_bunches):
        (ca, sa), (cb, sb) = a.download(j), b.download(j)
        assert np.array_equal(ca, cb) and np.array_equal(sa, sb)
        assert a.moments()[j].transmission == t[j]


def _bins(wl, z):
    """First and last bin that a particle is in (MPBunch.cpp:2052, 2170)."""
    r, t = wl.cfg.ring, wl.bbi_table
    if wl.cfg.bbi.time_domain:
        dz, lo = abs(t[1, 0] - t[0, 0]), -r.t0 * 299792458.0 / r.harmonics / 2
    else:
        dz = 1 / (2 * t[-1, 0]) * 299792458.0 * r.r_beta
        lo = -dz * (len(t) - 1) - dz / 2
    b = ((z - lo) / dz).astype(int)
    return b.min(), b.max()


@pytest.mark.parametrize("td,stretch,rows", CASES)
def test_potentials_on_every_bin_between_the_particles(td, stretch, rows):
    """The bins come from the particles, so that a bin or a plane left out
    shows."""
    wl, parts = _train(SIZES, stretch, td, rows)
    g, o = pair(wl, parts)
    for b in (g, o):
        b.BBImpBeamInteraction()
    for j, p in enumerate(parts):
        first, last = _bins(wl, p[4])
        a, have = g.bbi_profile(j)
        have = have[1:, first - a:last + 1 - a]
        want = o.bbi_profile(j)[1:, first:last + 1]
        assert have.shape == want.shape == (5, last + 1 - first)
        for q in range(5):
            k = np.max(np.abs(want[q]))
            assert k > 0 or p.shape[1] == 1  # one particle: its own wake can underflow
            assert np.max(np.abs(have[q] - want[q])) <= 1e-11 * k


@pytest.mark.parametrize("td", [0, 1])
@pytest.mark.parametrize("m", [148, 149])
def test_potentials_of_trains_round_the_smaller_convolutions(m, td):
    """More bunches than SMs take the convolution of 256 threads."""
    wl = configs.make("batched_uneven", n_scale=0.004)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:m].copy(), wl.harm[:m].copy(), wl.ne[:m].copy()
    c = wl.cfg
    c.flag_beam_ion = c.flag_lr_wake = c.flag_fir = c.flag_sr_wake = 0
    wl.set_bbi(bbicases.wake_table(400, 0.5e-3, 40) if td else bbicases.resonator_table(640, 300e9), td)
    parts = particles(wl, seed=19)
    g, o = pair(wl, parts)
    for b in (g, o):
        b.BBImpBeamInteraction()
    for j, p in enumerate(parts):
        first, last = _bins(wl, p[4])
        a, have = g.bbi_profile(j)
        have = have[:, first - a:last + 1 - a]
        want = o.bbi_profile(j)[:, first:last + 1]
        for q in range(6):
            assert np.max(np.abs(have[q] - want[q])) <= 1e-11 * np.max(np.abs(want[q]))
