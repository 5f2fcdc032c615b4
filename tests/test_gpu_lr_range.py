"""The long-range wake refuses centroids whose lags lie outside its table,
however far."""
import numpy as np
import pytest

from cetasim_b200 import _abi
from cetasim_b200.beam import MPBeam
from helpers import particles, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("z", [1e3, -1e3, 1e30, -1e30, 1e200, -1e200, np.inf, -np.inf, np.nan])
def test_lags_outside_the_table(z):
    wl = small("batched_uneven", 0.002, flag_beam_ion=0, flag_fir=0)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:3].copy(), wl.harm[:3].copy(), wl.ne[:3].copy()
    parts = particles(wl, seed=2)
    b = MPBeam(wl)
    for j, c in enumerate(parts):
        if j == 1:
            c[4] = z
        b.upload(j, c)
    b.MPBeamRMSCal(0)
    with pytest.raises(_abi.CgError, match="long-range wake lag outside"):
        b.LRWakeBeamIntaction()
    # the device goes on: the same train where it belongs
    for j, c in enumerate(particles(wl, seed=2)):
        b.upload(j, c)
    fresh = MPBeam(wl)
    for j, c in enumerate(particles(wl, seed=2)):
        fresh.upload(j, c)
    fresh.Run(0, 1)
    assert all(np.all(np.isfinite(fresh.download(j)[0])) for j in range(3))
