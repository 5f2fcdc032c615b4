"""Space charge at the edges of its kernels' sizes: meshes that end inside an
8 x 8 tile of the solve (2 x 2 to 64 x 64), slices up to and beyond the number
that a CTA keeps in shared memory, bunches that end inside a tile or a chunk
or have fewer particles than slices; one step against the oracle.
Tolerances: 1e-11 of the largest kick as for the reference's runs.  With more
slices than particles a slice of two particles r apart has sizes from sums
about the bunch's centroid, an error of 2^-52 (sigma / r)^2; among some
hundred such slices r > 1e-4 sigma but for one case in fifty: 1e-7."""
import numpy as np
import pytest

import oracle
from cetasim_b200 import configs
from cetasim_b200.beam import MPBeam
from helpers import particles

pytestmark = pytest.mark.gpu


def _step(flag, mesh, sizes, tol):
    wl = configs.make("fast_ion", n_scale=0.01)
    m = len(sizes)
    wl.n_macro, wl.harm, wl.ne = wl.n_macro[:m].copy(), wl.harm[:m].copy(), wl.ne[:m].copy()
    wl.n_macro[:] = sizes
    c = wl.cfg
    c.flag_beam_ion = c.flag_lr_wake = c.flag_fir = c.flag_sr_wake = 0
    c.flag_sc = flag
    c.sc_mesh[:] = mesh
    parts = particles(wl, seed=31, spread=1.0)
    got = []
    for cls in (oracle.OracleBeam, MPBeam):
        b = cls(wl)
        for j, p in enumerate(parts):
            b.upload(j, p)
        b.MPBeamRMSCal(0)
        b.BeamTransferDueToSpaceCharge(0)
        got.append([b.download(j)[0] for j in range(m)])
    for p, want, have in zip(parts, *got):
        assert np.array_equal(have[[0, 2, 4, 5]], p[[0, 2, 4, 5]])
        for q in (1, 3):
            k = np.max(np.abs(want[q] - p[q]))  # 0: no slice of two particles
            assert np.max(np.abs(have[q] - want[q])) <= tol * k


@pytest.mark.parametrize("mesh", [(2, 2, 2), (3, 33, 7), (8, 8, 1024), (9, 7, 1025), (31, 40, 11),
                                  (64, 64, 5), (64, 2, 3)])
def test_pic(mesh):
    _step(2, mesh, [2047, 2049, 33, 700, 17000], 1e-11)


@pytest.mark.parametrize("flag", [1, 3])
@pytest.mark.parametrize("nz", [2, 3, 33])
def test_slice_models(flag, nz):
    _step(flag, (32, 32, nz), [4097, 255, 30001], 1e-11 if nz < 4 else 1e-7)


@pytest.mark.parametrize("nz", [1024, 1025])
def test_linear_model_with_many_slices(nz):
    _step(3, (32, 32, nz), [2049, 700, 9000], 1e-7)
