"""The turn's tail where its kernels change path: RF phases at the quadrants'
edges and beyond the short argument reduction (against 80 bits), positions on
the loss limits and on the line below which no division is taken, and bunches
that end inside a warp or a tile (against the oracle and the staged calls)."""
import numpy as np
import pytest

from cetasim_b200.beam import MPBeam
from helpers import pair, particles, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 255, 257])
def test_rf_phases(n):
    """Tolerance: two ulps of the sine and cosine and one of the sum, of the
    voltage over the energy: 8 x 2^-53, and the rounding of the momentum."""
    wl = small("plain_single", n / 1e5)
    wl.n_macro[0] = n
    r = wl.cfg.ring
    theta = 2 * np.pi * r.cav_harm[0] * r.f0 * r.harmonics / (299792458.0 * r.r_beta)
    c = particles(wl, seed=3)[0]
    quarter = np.pi / 4 * np.arange(n)
    c[4] = np.where(np.arange(n) % 3 == 0, quarter, np.where(np.arange(n) % 3 == 1, -np.nextafter(quarter, 9e9),
                                                             1e5 + 7e3 * np.arange(n))) / theta
    c[5] = 0
    # the phase as the library rounds it (the coefficient in its order of
    # operations), its sine and cosine in 80 bits
    coeff = 1.0 / 299792458.0 / r.r_beta * 2.0 * np.pi * float(r.cav_harm[0]) * (r.f0 * r.harmonics)
    th = (c[4] * coeff).astype(np.longdouble)
    unit = 1.0 / np.longdouble(r.electron_energy) / np.longdouble(r.r_beta)**2
    want = (r.cav_vreq_re[0] * np.cos(th) + r.cav_vreq_im[0] * np.sin(th)) * unit
    g = MPBeam(wl)
    g.upload(0, c)
    g.BeamMomtumUpdateDueToRFTest()
    got = g.download(0)[0]
    assert np.array_equal(got[:5], c[:5])
    assert np.max(np.abs(got[5] - want)) <= 8 * 2.0**-53 * r.cav_vol[0] * unit


@pytest.mark.parametrize("n", [1, 31, 256, 300])
def test_loss_limits(n):
    """Marks and transmission are whole numbers: equal to the oracle's."""
    wl = small("plain_single", n / 1e5)
    wl.n_macro[0] = n
    s = wl.sections[0]
    r = wl.cfg.ring
    z_loss = r.t0 * 299792458.0 / r.harmonics / 2
    c = particles(wl, seed=5)[0]
    edge = [np.nextafter(1.0, 0), 1.0, np.nextafter(1.0, 2), np.sqrt(0.999), 1.1]
    for i in range(1, n):
        e = edge[i % 5] * (-1) ** i
        if i % 3 == 0:
            c[0, i], c[2, i] = e * s.aperture_x, 0.0
        elif i % 3 == 1:
            c[0, i], c[2, i] = 0.6 * e * s.aperture_x, 0.8 * e * s.aperture_y
        elif i % 4 == 0:
            c[4, i] = e * z_loss
    g, o = pair(wl, [c])
    tg, to = g.MarkParticleLostInBunch(), o.MarkParticleLostInBunch()
    assert np.array_equal(np.asarray(tg), np.asarray(to))
    assert np.array_equal(g.download(0)[1], o.download(0)[1])


@pytest.mark.parametrize("lost", ["x", "z"])
@pytest.mark.parametrize("config", ["plain_single", "fast_ion"])
def test_turn_ends_with_the_marks(config, lost):
    """A turn without wakes and feedback marks in the longitudinal pass: the
    turn equals its staged calls bit for bit, some particles lost."""
    over = {"flag_lr_wake": 0, "flag_sr_wake": 0, "flag_fir": 0, "flag_beam_ion": 0}
    wl = small(config, 0.01, **over)
    parts = particles(wl, seed=11)
    s, r = wl.sections[0], wl.cfg.ring
    z_loss = r.t0 * 299792458.0 / r.harmonics / 2
    for c in parts:
        if lost == "x":  # back inside at the turn's end
            c[0, ::7] += 1.01 * s.aperture_x
        else:
            c[4, ::7] += 1.01 * z_loss
    a, _ = pair(wl, parts)
    b, _ = pair(wl, parts)
    a.Run(0, 1)
    for k in range(wl.cfg.n_sections):
        b.BeamTransferPerInteractionPointDueToLatticeT(k)
    b.BeamMomtumUpdateDueToRFTest()
    b.BeamLongiPosTransferOneTurn()
    b.BeamEnergyLossOneTurn()
    b.BeamSynRadDamping(0)
    t = np.asarray(b.MarkParticleLostInBunch())
    for j in range(wl.n_bunches):
        (ca, sa), (cb, sb) = a.download(j), b.download(j)
        assert np.array_equal(ca, cb) and np.array_equal(sa, sb)
        assert a.moments()[j].transmission == t[j]
    assert lost == "x" or t.max() < 1


@pytest.mark.parametrize("config,scale", [("batched_uneven", 0.01), ("large_trapping", 0.005)])
def test_last_map_joins_the_tail_before_the_feedback(config, scale):
    """Turns with the feedback alone, whose last map is in the longitudinal
    pass: equal to their staged calls bit for bit."""
    wl = small(config, scale, flag_lr_wake=0, flag_sr_wake=0, flag_beam_ion=0, flag_fir=1)
    parts = particles(wl, seed=12)
    a, b = MPBeam(wl), MPBeam(wl)
    for j, c in enumerate(parts):
        a.upload(j, c)
        b.upload(j, c)
    a.Run(0, 3)
    for turn in range(3):
        for k in range(wl.cfg.n_sections):
            b.BeamTransferPerInteractionPointDueToLatticeT(k)
        b.BeamMomtumUpdateDueToRFTest()
        b.BeamLongiPosTransferOneTurn()
        b.BeamEnergyLossOneTurn()
        b.BeamSynRadDamping(turn)
        b.MPBeamRMSCal(0)
        b.FIRBunchByBunchFeedback(turn)
        b.MarkParticleLostInBunch()
    for j in range(wl.n_bunches):
        (ca, sa), (cb, sb) = a.download(j), b.download(j)
        assert np.array_equal(ca, cb) and np.array_equal(sa, sb)
