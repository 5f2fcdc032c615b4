"""The number of kernels that one turn launches, against the launches counted
by hand from the turn's stages."""
import ctypes as C

import pytest

import bbicases
from cetasim_b200 import configs
from cetasim_b200.beam import MPBeam

pytestmark = pytest.mark.gpu

# the wakes of one bunch: pass and merge, longitudinal, bins, potentials, kick, end
SINGLE = 7
# 20 sections of the ion train: moments (2), prep, walk, records, compact, pass
# each, a merge between sections, longitudinal, end
IONS = 2 + 20 * 5 + 19 + 2


def _launches(wl, prepare=None):
    b = MPBeam(wl)
    b.generate(5)
    if prepare:
        prepare(b)
    n = C.c_int()
    counts = []
    for _ in range(2):  # before and after the turn has run
        b._check(b.lib.cg_turn_launches(b.h, C.byref(n)))
        counts.append(n.value)
        b.Run(0, 1)
    assert counts[0] == counts[1]
    return counts[0]


def test_single_bunch():
    assert _launches(configs.make("plain_single", n_scale=0.05)) == SINGLE


@pytest.mark.parametrize("segments", [1, 2, 3])
def test_ion_train(segments):
    wl = configs.make("fast_ion", n_scale=0.02, bunch_current=2e-5)
    # each segment more is a walk, records and a pass more at every section
    want = IONS + 20 * 3 * (segments - 1)
    assert _launches(wl, lambda b: b.set_pipeline(segments)) == want


def test_ion_train_with_kick_and_map_apart():
    wl = configs.make("fast_ion", n_scale=0.02, bunch_current=2e-5)
    # a kick at every section; the last map joins the longitudinal pass
    assert _launches(wl, lambda b: b.set_kick_variant(0)) == IONS + 20 - 1


def _plain(**flags):
    wl = configs.make("fast_ion", n_scale=0.02)
    c = wl.cfg
    c.flag_beam_ion = c.flag_lr_wake = c.flag_fir = c.flag_sr_wake = 0
    for k, v in flags.items():
        setattr(c, k, v)
    return wl


# 20 sections: range (slice models), geometry, count, then offsets, scatter and
# solve or the slices, kick; passes and merges but for the last section, whose
# map joins the longitudinal pass; moments (2), longitudinal, end
@pytest.mark.parametrize("flag,each", [(1, 5), (2, 6), (3, 5)])
def test_space_charge(flag, each):
    wl = _plain(flag_sc=flag)
    wl.cfg.sc_mesh[:] = (16, 16, 9)
    assert _launches(wl) == 2 + 20 * each + 2 * 19 + 2


def test_impedance():
    # 19 maps, longitudinal with the last, histogram, convolution, kick, end
    wl = _plain()
    wl.set_bbi(bbicases.resonator_table(640, 300e9), 0)
    assert _launches(wl) == 19 + 1 + 3 + 1


def test_no_beam():
    b = MPBeam(configs.make("plain_single", n_scale=0.05))
    h, n = C.c_void_p(), C.c_int(-1)
    b._check(b.lib.cg_create(C.byref(b.wl.cfg), 0, C.byref(h)))
    assert b.lib.cg_turn_launches(h, C.byref(n)) == 0 and n.value == 0
    b.lib.cg_destroy(h)
