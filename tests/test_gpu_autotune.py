"""The autotuner times each kernel once: choices that run the same kernel share
a figure, and a switch without effect is left as it was."""
import pytest

from cetasim_b200.beam import MPBeam
from helpers import TRAPPED, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("switch", [False, True])
def test_choices_of_one_kernel_share_a_figure(switch):
    b = MPBeam(small("fast_ion", 0.05, bunch_current=TRAPPED))
    b.generate(3)
    b.Run(0, 1)
    b.set_map_async(switch)
    choice, ms = b.autotune(0, reps=3)
    n = len(ms) - 4
    assert n == 8 and ms[0] == ms[1] == ms[4] == ms[7] and ms[3] == ms[5] == ms[6]
    assert choice % n in (0, 2, 3)  # the first choice of each kernel
    assert ms[n] == ms[n + 2] and ms[n + 1] == ms[n + 3]
    assert b.map_async() == switch
