"""Particles with a coordinate that is not finite in a ring without dispersion,
whose maps leave out the matrices' zeros: their z is no number either, as with
the zeros, and the stages that look at z refuse the turn."""
import numpy as np
import pytest

from cetasim_b200 import _abi, configs
from cetasim_b200.beam import MPBeam
from helpers import particles, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage", ["map", "damping"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_z_follows_the_transverse_coordinates(bad, stage):
    wl = small("plain_single", 0.003)
    clean = particles(wl, seed=4)[0]
    parts = clean.copy()
    for q in range(4):
        parts[q, 10 + 64 * q] = bad
    hit = np.zeros(parts.shape[1], dtype=bool)
    hit[10:10 + 64 * 4:64] = True
    out = []
    for c in (clean, parts):
        b = MPBeam(wl)
        b.upload(0, c)
        if stage == "map":
            b.BeamTransferPerInteractionPointDueToLatticeT(0)
        else:
            b.BeamSynRadDamping(0)
        out.append(b.download(0)[0])
    assert np.array_equal(out[0][:, ~hit], out[1][:, ~hit])
    assert np.all(np.isnan(out[1][4, hit])) and np.all(np.isfinite(out[1][5, hit]))


def test_bunches_of_one_particle_in_an_ion_train_are_refused():
    """Their size is zero, so the ions' field is no number, and the long-range
    wake refuses the bunches' centroids."""
    wl = configs.make("batched_uneven", n_scale=1e-6, bunch_current=2e-6)
    b = MPBeam(wl)
    b.generate(7)
    with pytest.raises(_abi.CgError):
        b.Run(0, 1)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_damping_with_a_momentum_that_is_not_finite(bad):
    """The damping's zeros bring it into every coordinate."""
    wl = small("plain_single", 0.003)
    c = particles(wl, seed=4)[0]
    c[5, 17] = bad
    b = MPBeam(wl)
    b.upload(0, c)
    b.BeamSynRadDamping(0)
    got = b.download(0)[0]
    assert np.all(np.isnan(got[:5, 17])) and not np.isfinite(got[5, 17])
    assert np.all(np.isfinite(np.delete(got, 17, axis=1)))
