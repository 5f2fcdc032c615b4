"""The slice of a particle at the limits of its longitudinal position."""
import numpy as np
import pytest

import oracle
from cetasim_b200 import configs
from cetasim_b200.beam import MPBeam
from helpers import particles

pytestmark = pytest.mark.gpu


def _train(flag, mesh, sizes):
    wl = configs.make("fast_ion", n_scale=0.01)
    m = len(sizes)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:m].copy(), wl.harm[:m].copy(), wl.ne[:m].copy()
    wl.n_macro[:] = sizes
    c = wl.cfg
    c.flag_beam_ion = c.flag_lr_wake = c.flag_fir = c.flag_sr_wake = 0
    c.flag_sc = flag
    c.sc_mesh[:] = mesh
    return wl, particles(wl, seed=31, spread=1.0)


def _kick(wl, parts, surv, cls=MPBeam):
    b = cls(wl)
    for j, p in enumerate(parts):
        b.upload(j, p, surv[j])
    b.MPBeamRMSCal(0)
    b.BeamTransferDueToSpaceCharge(0)
    return [b.download(j)[0] for j in range(len(parts))]


@pytest.mark.parametrize("nz", [7, 1100])
@pytest.mark.parametrize("flag", [1, 2, 3])
def test_a_position_that_is_no_number_is_in_the_first_slice(flag, nz):
    """Bit for bit the kicks of the same beam with those (lost) particles ahead
    of the first slice."""
    wl, parts = _train(flag, (9, 8, nz), [2049, 700])
    surv = [np.zeros(p.shape[1], dtype=np.uint8) for p in parts]
    got = []
    for z in (np.nan, -1.0):
        for p, s in zip(parts, surv):
            p[4, 5::300], s[5::300] = z, 2
        got.append(_kick(wl, parts, surv))
    for a, b in zip(*got):
        assert np.array_equal(a[:4], b[:4], equal_nan=True) and np.array_equal(a[5], b[5])


@pytest.mark.parametrize("flag", [1, 2, 3])
def test_infinite_positions_are_in_the_outer_slices(flag):
    """Likewise for lost particles infinitely far ahead and behind."""
    wl, parts = _train(flag, (9, 8, 7), [2049, 700])
    surv = [np.zeros(p.shape[1], dtype=np.uint8) for p in parts]
    got = []
    for z in (np.inf, 1.0):
        for p, s in zip(parts, surv):
            p[4, 5::300], s[5::300] = z, 2
            p[4, 6::300], s[6::300] = -z, 2
        got.append(_kick(wl, parts, surv))
    for a, b in zip(*got):
        assert np.array_equal(a[:4], b[:4], equal_nan=True) and np.array_equal(a[5], b[5])


@pytest.mark.parametrize("flag,nz", [(1, 33), (2, 33), (2, 100), (3, 33)])
def test_positions_on_the_edges_of_slices(flag, nz):
    """Particles at the slices' edges, where the quotient (z - zMin) / dz is a
    whole number or just below one, against the oracle's slices.  Tolerance:
    1e-11 of the largest kick as for the reference's runs; a particle in the
    neighbouring slice changes the kicks of some hundred by a hundredth."""
    wl, parts = _train(flag, (9, 8, nz), [6000, 9000])
    rng = np.random.default_rng(3)
    moved = 0
    for p in parts:
        p[4] = rng.uniform(-6e-3, 5.7e-3, p.shape[1])
        z0, z1 = p[4].min() - 1e-6, p[4].max() + 1e-6
        dz = (z1 - z0) / (nz - 1)
        edge = z0 + np.arange(1, nz - 1) * dz
        inner = np.flatnonzero((p[4] > p[4].min()) & (p[4] < p[4].max()))[:2 * len(edge)]
        p[4, inner] = np.concatenate([edge, np.nextafter(edge, -1)])
        s = p[4] - z0
        moved += np.count_nonzero(np.floor(s * (1 / dz)) != np.floor(s / dz))
    assert moved > 0  # the case is one that a product with 1 / dz would get wrong
    surv = [np.zeros(p.shape[1], dtype=np.uint8) for p in parts]
    for p, want, have in zip(parts, *(_kick(wl, parts, surv, c) for c in (oracle.OracleBeam, MPBeam))):
        for q in (1, 3):
            k = np.max(np.abs(want[q] - p[q]))
            assert np.max(np.abs(have[q] - want[q])) <= 1e-11 * k


@pytest.mark.parametrize("flag", [1, 2])
def test_chunks_of_more_tiles_than_one_round(flag):
    """A bunch of more than 256 chunks of eight tiles, beside a small one,
    against the oracle; tolerance as for the edges."""
    wl, parts = _train(flag, (9, 8, 5), [531000, 700])
    surv = [np.zeros(p.shape[1], dtype=np.uint8) for p in parts]
    for p, want, have in zip(parts, *(_kick(wl, parts, surv, c) for c in (oracle.OracleBeam, MPBeam))):
        for q in (1, 3):
            k = np.max(np.abs(want[q] - p[q]))
            assert np.max(np.abs(have[q] - want[q])) <= 1e-11 * k
