"""The training kernel at one tile, an odd number of tiles and more tiles than
SMs: loss and gradients against the FP64 network, with the tolerances of the
512-sample test (1e-6 of the loss, 1e-4 of each layer's gradient)."""
import numpy as np
import pytest

from cetasim_b200 import surrogate as S
from oracle import mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 384, 128 * 149])
def test_gradients(n):
    w = mlp.init(9)
    x, t = S.dataset(11, n)
    loss, g = S.gradient(w, x, t)
    lref, gref = mlp.loss_and_grad(w, x, t)
    assert abs(loss - lref) <= 1e-6 * lref
    for o, k in ((mlp.W1, 192), (mlp.B1, 64), (mlp.W2, 4096), (mlp.B2, 64), (mlp.W3, 4096),
                 (mlp.B3, 64), (mlp.W4, 128), (mlp.B4, 2)):
        assert np.linalg.norm(g[o:o + k] - gref[o:o + k]) <= 1e-4 * np.linalg.norm(gref[o:o + k])
    again = S.gradient(w, x, t)
    assert again[0] == loss and np.array_equal(again[1], g)


def test_gradients_of_two_threads():
    """Calls from two host threads share the pool of device memory: each gets
    the gradient that it gets alone, bit for bit."""
    from concurrent.futures import ThreadPoolExecutor
    n = (128 * 9, 128)
    args = [(mlp.init(9 + i), *S.dataset(11 + i, n[i])) for i in range(2)]
    alone = [S.gradient(*a) for a in args]
    with ThreadPoolExecutor(2) as ex:
        both = list(ex.map(lambda i: (i, S.gradient(*args[i])), [0, 1] * 20))
    for i, (loss, grad) in both:
        assert loss == alone[i][0] and np.array_equal(grad, alone[i][1])
