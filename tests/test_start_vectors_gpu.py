"""Gaussian start vectors drawn on the GPU (k_start_gauss) against the oracle's
libstdc++ sequence (main.cpp:1015-1025): Lanczos from the engine's own start
vectors and from the oracle's, in FP64, on blocks of 1 row to several thousand,
below, at and above the 156 pairs that one state of the generator yields.

The vectors differ by the rounding of the logarithm and of the norm (about
4 x 2^-53 per element), which the first 4 steps of these blocks amplify by less
than 1e3: 1e-12 relative.
"""
import numpy as np
import pytest

import pyoracle as O

import ftlm_extended_hubbard_development_b200 as pkg

pytestmark = pytest.mark.gpu

# lx, ly, N_up, N_down, mx, my: dimensions 1 to 10^4
BLOCKS = [(2, 2, 0, 0, 0, 0), (2, 2, 2, 2, 0, 0), (3, 2, 3, 3, 1, 0), (4, 2, 2, 4, 0, 0), (4, 2, 4, 4, 0, 0),
          (3, 3, 4, 4, 1, 2), (4, 3, 4, 5, 0, 0), (4, 3, 5, 5, 3, 1)]


@pytest.mark.parametrize("block", BLOCKS, ids=lambda b: "%dx%d_%d_%d_k%d%d" % b)
def test_start_vectors_match_the_oracle(block):
    lx, ly, nu, nd, mx, my = block
    m = pkg.Model(lx=lx, ly=ly, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)
    dim = O.block_csr(O.Model(**m.__dict__), nu, nd, mx, my).dim
    samples, steps = 3, min(4, dim)
    seed = O.block_seed(12345, nu, nd, mx, my)
    starts = np.stack([O.start_vector(seed, s, dim) for s in range(samples)])
    opts = pkg.RunOpts(samples=samples, lanczos_steps=steps, exact_block_threshold=0)
    with pkg.Engine(m, opts) as eng:
        eng.sector_prepare(nu, nd)
        a, b, s = eng.block_lanczos(mx, my)
        ra, rb, rs = eng.block_lanczos(mx, my, start=starts)
        assert np.array_equal(s, rs)
        size = max(1.0, np.abs(ra).max())
        assert np.abs(a - ra).max() <= 1e-12 * size
        assert np.abs(b - rb).max() <= 1e-12 * size
        # the same vectors in the launch of all small blocks
        eng.blocks_ftlm_batched([(mx, my)])
        ev, w, _ = eng.block_spectrum(mx, my, exact=False)
    with pkg.Engine(m, opts) as eng:
        eng.sector_prepare(nu, nd)
        ev2, w2, _ = eng.block_spectrum(mx, my, exact=False)
    assert np.abs(ev - ev2).max() <= 1e-10 * size and np.abs(w - w2).max() <= 1e-10
