"""The slice of a particle at the limits of its longitudinal position."""
import numpy as np
import pytest

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


def _kick(wl, parts, surv):
    b = MPBeam(wl)
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
