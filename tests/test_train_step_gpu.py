"""The two-launch training step (k_train_rows, k_train_params) at the sizes where
its tiling can go wrong: layers narrower than a warp and not a multiple of 4,
wider than the CTA, batches below, at and above the rows a CTA takes, and
parameters that no longer fit in shared memory (the per-layer kernels), against
the FP64 oracle.

Bounds. One Adam step from zero moments moves a parameter by
lr g / (|g| + eps); an error dg of the gradient moves that by at most
lr min(2, dg / |g|). A gradient is a sum over the batch of products through the
layers: dg <= 2^-24 (batch + sum of widths + 16) G with G the largest gradient
of the same layer kind, the oracle's largest absolute entry times 8. The loss is
a mean of squares: 1e-5 relative.
"""
import numpy as np
import pytest

import mlp_oracle as O

from ftlm_extended_hubbard_development_b200.engine import Mlp

pytestmark = pytest.mark.gpu

# n_in, width, depth, n_out, batch
SIZES = [(1, 1, 1, 1, 1), (3, 5, 1, 2, 3), (20, 128, 3, 32, 128), (33, 128, 3, 32, 149), (52, 128, 3, 32, 500),
         (32, 128, 3, 32, 512), (6, 30, 4, 33, 593), (32, 128, 3, 32, 1021), (7, 300, 1, 3, 70),
         (16, 256, 3, 8, 64)]  # the last does not fit


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%d_%dx%d_%d_b%d" % s)
def test_one_step_against_the_oracle(size):
    n_in, width, depth, n_out, batch = size
    rng = np.random.default_rng(7)
    x = rng.standard_normal((batch, n_in)).astype(np.float32)
    t = rng.standard_normal((batch, n_out)).astype(np.float32)
    mask = (0.05 + rng.random((batch, n_out))).astype(np.float32)
    shapes = O.layer_shapes(n_in, width, depth, n_out)
    p0 = np.concatenate([np.concatenate([rng.uniform(-1, 1, i * o) * np.sqrt(6.0 / (i + o)), 0.1 * rng.standard_normal(o)])
                         for i, o in shapes]).astype(np.float32)
    lr = 1e-2
    net = Mlp(n_in, width, depth, n_out)
    net.set_params(p0)
    hist = net.train(x, t, mask, 1, batch, lr)
    got = net.get_params()
    net.close()
    loss, g = O.loss_grad(p0, shapes, x, t, mask)
    want = O.adam_steps(p0, shapes, [(x, t, mask)], lr)
    assert abs(hist[0] - loss) <= 1e-5 * loss
    dg = 2.0 ** -24 * (batch + depth * width + n_in + 16) * 8.0 * np.abs(g).max()
    bound = lr * np.minimum(2.0, dg / np.maximum(np.abs(g), 1e-300)) + 2.0 ** -22 * (np.abs(p0) + lr)
    assert np.all(np.abs(got - want) <= bound), (np.abs(got - want) / bound).max()


def test_both_routes_give_the_same_bits():
    """A batch larger than the data is the data: its gradient by loss_grad (the
    per-layer kernels) and Adam's first step in FP32 give the parameters that
    the two-launch step leaves, up to the order of the rows in the batch."""
    rng = np.random.default_rng(3)
    n = 256
    x = rng.standard_normal((n, 20)).astype(np.float32)
    t = rng.standard_normal((n, 32)).astype(np.float32)
    mask = (0.05 + rng.random((n, 32))).astype(np.float32)
    x[:] = x[0]
    t[:] = t[0]
    mask[:] = mask[0]  # equal rows: any order is the same order
    a, b = Mlp(20, 128, 3, 32, seed=4), Mlp(20, 128, 3, 32, seed=4)
    p0 = a.get_params()
    loss, grad = a.loss_grad(x, t, mask)
    hist = b.train(x, t, mask, 1, n, 1e-3)
    got = b.get_params()
    a.close()
    b.close()
    f = np.float32
    m, v = (f(1) - f(0.9)) * grad, (f(1) - f(0.999)) * grad * grad
    c1, c2 = f(1) - f(0.9), f(1) - f(0.999)
    want = p0 - f(1e-3) * (m / c1) / (np.sqrt(v / c2) + f(1e-8))
    assert hist[0] == loss
    # Adam in numpy rounds every operation, the kernel fuses some: 8 u of the step, u of the parameter
    assert np.all(np.abs(got - want) <= 2.0 ** -21 * 1e-3 + 2.0 ** -23 * np.abs(p0))
