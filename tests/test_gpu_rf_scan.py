"""The scans of the beam-loading recurrence (k_rf_prep, k_rf_chain) against
the oracle's step-by-step recurrence, at the sizes where the scans change
shape: bins around the 64 of one scan tile, bunches around the 512 threads of
the train scan, gaps of one bucket and of thousands.  Tolerance: the 1e-12 of
the staged RF steps (both sides round each of at most 1e5 steps)."""
import tempfile

import numpy as np
import pytest

import blcases
import oracle
from cetasim_b200.beam import MPBeam
from helpers import particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bunches,bins,excite", [(1, 1, 1), (2, 64, 1), (5, 65, 1), (511, 33, 1),
                                                 (513, 2, 1), (900, 130, 1), (513, 40, 0)])
def test_rf_steps_match_the_sequential_recurrence(bunches, bins, excite):
    with tempfile.TemporaryDirectory() as d:
        wl, _, _ = blcases.build("ragged_harmonic", d)
    wl.n_macro, wl.harm, wl.ne = (a[:bunches].copy() for a in (wl.n_macro, wl.harm, wl.ne))
    wl.cfg.ring.rf_bunch_bins = bins
    wl.cfg.ring.res_excite[1] = excite
    parts = particles(wl, seed=3, spread=1.0)
    b, o = MPBeam(wl), oracle.OracleBeam(wl)
    for j, c in enumerate(parts):
        b.upload(j, c)
        o.upload(j, c)
    for _ in range(2):
        for x in (b, o):
            x.BeamMomtumUpdateDueToRFTest()
            x.BeamLongiPosTransferOneTurn()
    for j in range(bunches):
        got, s = b.download(j)
        want, _ = o.download(j)
        assert blcases.coord_rel_err(got, want, s == 0).max() <= 1e-12
    for x, y in zip(b.resonator(1), o.resonator(1)):
        assert abs(x - y) <= 1e-12 * (abs(y) + 1e-300)


def test_one_bin_of_infinite_width():
    """The head bin's voltage needs no rotation: the induced voltage of a bunch
    with a particle infinitely far away is that of the same bunch without."""
    with tempfile.TemporaryDirectory() as d:
        wl, _, _ = blcases.build("ragged_harmonic", d)
    wl.n_macro, wl.harm, wl.ne = (a[:1].copy() for a in (wl.n_macro, wl.harm, wl.ne))
    wl.cfg.ring.rf_bunch_bins = 1
    wl.cfg.ring.res_excite[1] = 1
    parts = particles(wl, seed=3, spread=1.0)[0]
    induced = []
    for z in (parts[4, 1], np.inf):
        parts[4, 1] = z
        b = MPBeam(wl)
        b.upload(0, parts)
        b.BeamMomtumUpdateDueToRFTest()
        induced.append(b.rf_info(0, 1)[2])
    assert np.isfinite(induced[0]) and induced[0] == induced[1]
