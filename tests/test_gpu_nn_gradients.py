"""Weight, bias and input gradients of the warm-start network (the
transposed im2col, bias sums, split-K sums and col2im kernels of
agdeblend_b200/csrc/nn_kernels.cuh and tc_gemm.cuh) against the float64
oracle at sizes where they take their other paths: image rows that are not a
multiple of eight pixels on the lower levels (8, 4, 2, 1), pixel counts below,
at and above a bias chunk (8192), one input channel and three, channel counts
with and without a factor four.

Every value that is rounded to BF16 on the way is exact before it is rounded,
so the GPU and the oracle round the same numbers: weights are one +-1 per
output channel, biases zero, inputs and targets multiples of 64, the pixel
count (the loss's divisor) a power of two.  What is left is the FP32 sum of
at most 2^15 products per weight, in blocks: 1e-5 relative L2."""
import numpy as np
import pytest

import nn_oracle as N
from agdeblend_b200.nn import WarmStartNet
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _params(base, in_ch, rng):
    parts = []
    for cin, cout, _ in N.architecture(base, in_ch)[0]:
        w = np.zeros((cout, 9 * cin), np.float32)
        w[np.arange(cout), rng.integers(0, 9 * cin, cout)] = rng.choice([-1.0, 1.0, 1.0], cout)
        parts += [w.reshape(-1), np.zeros(cout, np.float32)]
    return np.concatenate(parts)


@pytest.mark.parametrize("base,n,h,w,in_ch", [(4, 8, 8, 8, 1), (4, 16, 8, 16, 3),
                                              (6, 8, 8, 32, 1), (4, 8, 32, 32, 1),
                                              (8, 4, 64, 64, 3), (4, 8, 64, 64, 1)])
def test_gradients_match_oracle(base, n, h, w, in_ch):
    net = WarmStartNet(base, seed=1, in_channels=in_ch)
    rng = np.random.default_rng(n * h * w)
    p = _params(base, in_ch, rng)
    net.set_params(p)
    shape = (n, h, w) if in_ch == 1 else (n, h, w, in_ch)
    x = (64 * rng.integers(-2, 3, shape)).astype(np.float32)
    t = (64 * rng.integers(-2, 3, (n, h, w))).astype(np.float32)
    loss_o, g_o = N.Net(base, p.astype(np.float64), bf16_like_gpu=True, in_ch=in_ch).loss_grad(
        x.astype(np.float64), t.astype(np.float64))
    loss, g = net.loss_grad(x, t)
    assert np.linalg.norm(g_o) > 0
    assert abs(loss - loss_o) <= 1e-5 * loss_o
    assert rel_l2(g, g_o) <= 1e-5
    net.close()
