"""The walk's branches against the oracle at the sizes where they change:
train lengths around the 16 steps of a window, clouds below and above the
18944 trajectories from which one lane walks a whole ion, horizontal,
vertical, round and mixed bunches, ions outside the loss bounds and beyond
|z| = 30.  Tolerance 1e-11 as in the other chain tests (a few passages at a
current where the ions are trapped)."""
import numpy as np
import pytest

from cetasim_b200 import configs
from helpers import TRAPPED, particles, small
import oracle
from cetasim_b200.beam import MPBeam

pytestmark = pytest.mark.gpu


def _shape(parts, kind):
    for j, c in enumerate(parts):
        k = kind if kind != "mixed" else ("flat", "tall", "round")[j % 3]
        if k == "tall":
            c[[0, 2]], c[[1, 3]] = c[[2, 0]], c[[3, 1]]
        elif k == "round":
            c[2], c[3] = c[0], c[1]
    return parts


@pytest.mark.parametrize("bunches,ions,kind", [
    (1, 0, "flat"), (15, 100, "flat"), (16, 63, "tall"), (17, 65, "round"), (33, 1000, "mixed"),
    (4, 18944 - 4, "flat"), (4, 18944 - 3, "flat"), (17, 20000, "tall"), (9, 40001, "mixed"),
])
def test_walk_matches_the_oracle(bunches, ions, kind):
    wl = small("fast_ion", 0.02, bunch_current=TRAPPED)
    wl.n_macro, wl.harm, wl.ne = (a[:bunches].copy() for a in (wl.n_macro, wl.harm, wl.ne))
    parts = _shape(particles(wl, seed=4, spread=1.0), kind)
    g, o = MPBeam(wl), oracle.OracleBeam(wl)
    for j, c in enumerate(parts):
        g.upload(j, c)
        o.upload(j, c)
    if ions:
        x, y, vx, vy = configs.preload_clouds(wl, ions, seed=7)[0]
        x[::37] *= 60.0  # outside the loss bounds, some beyond |z| = 30
        for b in (g, o):
            b.upload_ions(0, 0, x, y, vx, vy)
    for turn in range(2):
        for b in (g, o):
            b.MPBeamRMSCal(0)
            b.SSBeamIonEffectOneInteractionPoint(turn, 0)
        rg, ro = g.cloud_record(0), o.cloud_record(0)
        assert np.array_equal(rg[..., 5], ro[..., 5])
        assert np.allclose(rg[..., :3], ro[..., :3], rtol=1e-11, atol=0)
        scale = np.maximum(ro[..., 1:3], 1e-300)
        assert np.all(np.abs(rg[..., 3:5] - ro[..., 3:5]) <= 1e-11 * scale)
        ig, io = g.ions(0), o.ions(0)
        assert len(ig[0]) == len(io[0])
        for a, b in zip(ig, io):
            if len(b):
                assert np.allclose(a, b, rtol=1e-11, atol=1e-11 * np.max(np.abs(b)))
