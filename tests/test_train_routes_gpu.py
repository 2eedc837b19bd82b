"""Training on the two-launch step against the per-layer kernels, which sum every
product in the same index order: equal bits in the parameters and in the loss of every
epoch. Distinct rows, several epochs and batches (so that batches start inside the
order of an epoch), batches that are no multiple of the 128 rows of a stage, a dropped
tail, and the 1, 2, 4 and 8 rows that a CTA takes."""
import numpy as np
import pytest

from ftlm_extended_hubbard_development_b200.engine import Mlp

pytestmark = pytest.mark.gpu


# n_in, width, depth, n_out, rows, batch
@pytest.mark.parametrize("size", [(20, 128, 3, 32, 500, 97), (32, 128, 3, 32, 1100, 256), (33, 64, 2, 7, 1300, 500),
                                  (52, 128, 3, 32, 2600, 1021), (3, 5, 1, 2, 50, 3)], ids=str)
def test_equal_bits(size, monkeypatch):
    n_in, width, depth, n_out, n, batch = size
    rng = np.random.default_rng(11)
    x = rng.standard_normal((n, n_in)).astype(np.float32)
    t = rng.standard_normal((n, n_out)).astype(np.float32)
    mask = ((rng.random((n, n_out)) < 0.8) * (0.05 + rng.random((n, n_out)))).astype(np.float32)
    out = []
    for step in ("", "layers"):
        monkeypatch.setenv("FTLM_TRAIN_STEP", step)
        net = Mlp(n_in, width, depth, n_out, seed=5)
        hist = net.train(x, t, mask, 3, batch, 3e-3, seed=17)
        out.append((np.asarray(hist).copy(), net.get_params()))
        net.close()
    assert np.all(np.isfinite(out[0][1]))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0])
