"""The warm start's network at the shapes where its products change form: widths that are no
multiple of four (element-wise staging), hidden widths beyond one slab of the inner dimension,
and batches large enough that a CTA takes two, four or sixteen row tiles.

Tolerances as in test_gpu_learned.py: FP32 against the FP64 oracle, outputs 1e-5, gradients 1e-4
(relative 2-norm)."""
import numpy as np
import pytest

import mlp_oracle as M
from femm_gpu_b200 import learned

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


def data(B, I, O, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(B, I)).astype(np.float32), rng.normal(size=(B, O)).astype(np.float32)


@pytest.mark.parametrize("I, H, O, B", [(4, 9, 3, 9600), (4, 16, 33, 4800), (3, 33, 5, 9601), (4, 64, 7, 20000),
                                        (4, 65, 96, 2401), (4, 128, 16, 4801), (4, 129, 16, 4801), (17, 30, 1, 40003)])
def test_large_batches_give_the_bits_of_small_ones(gpu, I, H, O, B):
    net = learned.Mlp(I, H, O, seed=3)
    x, _ = data(B, I, O, seed=B)
    y = net.forward(x)
    parts = np.concatenate([net.forward(x[i:i + 96]) for i in range(0, B, 96)])
    assert np.array_equal(y, parts)
    y64, _ = M.forward(net.get_parameters(), x, I, H, O)
    assert rel(y, y64) <= 1e-5


@pytest.mark.parametrize("I, H, O, B", [(4, 300, 50, 64), (5, 30, 7, 33), (3, 257, 1, 17), (4, 48, 8, 1), (1, 1, 1, 600),
                                        (4, 520, 96, 40), (4, 64, 8, 5000)])
def test_gradients_match_the_oracle(gpu, I, H, O, B):
    net = learned.Mlp(I, H, O, seed=5)
    p = net.get_parameters()
    x, t = data(B, I, O, seed=B)
    loss, g = net.loss_gradient(x, t)
    loss64, g64 = M.loss_gradient(p, x, t, I, H, O)
    assert abs(loss - loss64) <= 1e-5 * loss64
    o = 0
    for n in (H * I, H, H * H, H, O * H, O):
        assert rel(g[o:o + n], g64[o:o + n]) <= 1e-4, (o, n)
        o += n
