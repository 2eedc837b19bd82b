"""Blocks of small sectors (all tables of a sector in one launch, rows of many
blocks in one) against the oracle: every momentum block of sectors with one
segment, with two hops onto one target (lattices two sites wide), with empty
blocks, with 64-bit words, at the edges of the size classes of the small-block
Lanczos (512 / 1024 rows), and a sector whose tables are too many for the
sector-wide build (9x5, (0, 4): built block by block).

Exact spectra: both sides diagonalise in FP64 with backward-stable methods, so
an eigenvalue moves by at most p(n) u ||H||; n u ||H|| is used (||H|| bounded by
the largest absolute row sum). Lanczos coefficients of few steps: 1e-10, the
bound used for the sweep path before the reproducibility horizon.
"""
import numpy as np
import pytest

import pyoracle as O

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

pytestmark = pytest.mark.gpu

SECTORS = [(2, 2, 1, 1), (2, 2, 0, 3), (2, 2, 4, 4), (1, 5, 2, 2), (6, 1, 3, 3), (3, 2, 2, 4), (4, 2, 2, 2), (3, 3, 3, 1),
           (11, 3, 1, 1)]


def model(lx, ly):
    return pkg.Model(lx=lx, ly=ly, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)


@pytest.mark.parametrize("sector", SECTORS, ids=lambda s: "%dx%d_%d_%d" % s)
def test_exact_blocks_of_a_sector(sector):
    lx, ly, nu, nd = sector
    m = model(lx, ly)
    om = O.Model(**m.__dict__)
    with pkg.Engine(m) as eng:
        info = eng.sector_prepare(nu, nd)
        blocks = [(k % lx, k // lx) for k, d in enumerate(info.block_dims) if d > 0]
        eng.blocks_exact_batched(blocks)
        for mx, my in blocks:
            csr = O.block_csr(om, nu, nd, mx, my)
            ev, _, _ = eng.block_spectrum(mx, my, exact=True)
            rows = np.abs(csr.diag) + np.array([np.abs(csr.val[a:b]).sum() for a, b in
                                                zip(csr.row_ptr[:-1], csr.row_ptr[1:])])
            tol = csr.dim * 2.0 ** -53 * rows.max() * 4
            assert ev.shape == (csr.dim,)
            assert np.abs(ev - O.block_exact(csr)).max() <= max(tol, 1e-14), (mx, my)


# one size alone and several together: matrices of whole clusters (of 2, 4 and
# 8 CTAs) beside matrices of one CTA
@pytest.mark.parametrize("sector,count", [((3, 3, 2, 3), 1), ((3, 3, 2, 3), 9), ((4, 2, 3, 4), 3), ((4, 2, 2, 3), 8),
                                          ((3, 3, 3, 3), 2), ((3, 3, 3, 4), 1)],
                         ids=lambda x: "%dx%d_%d_%d" % x if isinstance(x, tuple) else "x%d" % x)
def test_dense_solver_by_clusters(sector, count):
    lx, ly, nu, nd = sector
    m = model(lx, ly)
    om = O.Model(**m.__dict__)
    with pkg.Engine(m) as eng:
        eng.spectra_defer(True)
        eng.sector_prepare(1, 1)  # small matrices in the same launch
        eng.blocks_exact_batched([(k % lx, k // lx) for k in range(lx * ly)])
        eng.sector_prepare(nu, nd)
        blocks = [(k % lx, k // lx) for k in range(count)]
        eng.blocks_exact_batched(blocks)
        for mx, my in blocks:
            csr = O.block_csr(om, nu, nd, mx, my)
            ev, _, _ = eng.block_spectrum(mx, my, exact=True)
            rows = np.abs(csr.diag) + np.add.reduceat(np.abs(csr.val), csr.row_ptr[:-1])
            assert np.all(np.diff(ev) >= 0)
            assert np.abs(ev - O.block_exact(csr)).max() <= csr.dim * 2.0 ** -53 * rows.max() * 4, (mx, my)
        eng.spectra_defer(False)


def test_dense_solver_with_work_vectors_in_global_memory():
    """4324 rows: three work vectors no longer fit in shared memory. Sum and
    sum of squares of the eigenvalues against trace and Frobenius norm."""
    m = model(7, 7)
    csr = O.block_csr(O.Model(**m.__dict__), 0, 4, 1, 2)
    with pkg.Engine(m) as eng:
        eng.sector_prepare(0, 4)
        ev, _, _ = eng.block_spectrum(1, 2, exact=True)
    assert len(ev) == csr.dim > 4266 and np.all(np.diff(ev) >= 0)
    row = np.repeat(np.arange(csr.dim), np.diff(csr.row_ptr))
    import scipy.sparse as sp
    h = sp.csr_matrix((csr.val, (row, csr.col)), shape=(csr.dim, csr.dim)) + sp.diags(csr.diag)
    norm = abs(h).sum(1).max()
    each = csr.dim * 2.0 ** -53 * norm  # per eigenvalue
    assert abs(ev.sum() - h.diagonal().real.sum()) <= csr.dim * each
    assert abs((ev ** 2).sum() - (abs(h).power(2)).sum()) <= 2 * csr.dim * norm * each


# dims around 512 and 1024, and one far above
FTLM = [(4, 2, 3, 4, 2, 0), (3, 3, 2, 5, 1, 1), (3, 3, 3, 3, 0, 0), (3, 3, 3, 4, 2, 2), (4, 3, 2, 4, 1, 2),
        (9, 5, 0, 4, 2, 1)]


@pytest.mark.parametrize("defer", [False, True], ids=["immediate", "pooled"])
@pytest.mark.parametrize("block", FTLM, ids=lambda b: "%dx%d_%d_%d_k%d%d" % b)
def test_small_lanczos_matches_the_oracle(block, defer):
    lx, ly, nu, nd, mx, my = block
    m = model(lx, ly)
    steps, R = 8, 3
    csr = O.block_csr(O.Model(**m.__dict__), nu, nd, mx, my)
    assert 256 < csr.dim <= 4096
    seed = O.block_seed(12345, nu, nd, mx, my)
    want = [O.tridiag_jacobi(*O.lanczos(csr, O.start_vector(seed, s, csr.dim), steps)) for s in range(R)]
    with pkg.Engine(m, pkg.RunOpts(samples=R, lanczos_steps=steps)) as eng:
        eng.thermo_configure([2.0], [0.0])
        eng.spectra_defer(defer)
        eng.sector_prepare(nu, nd)
        eng.blocks_ftlm_batched([(mx, my)])
        ev, w, pref = eng.block_spectrum(mx, my)
        eng.spectra_defer(False)
    e0 = np.concatenate([e for e, _ in want])
    assert pref == csr.dim
    assert np.abs(ev - e0).max() <= 1e-10 * max(1.0, np.abs(e0).max())
    w0 = np.concatenate([v for _, v in want]) / R
    assert np.abs(w - w0).max() <= 1e-8


def test_pooled_blocks_of_many_sectors_equal_the_immediate_ones():
    """Pool buffers grow (and move) while earlier sectors' Lanczos runs on the
    side streams; the spectra stay the same bits."""
    m = model(3, 3)
    opts = pkg.RunOpts(samples=4, lanczos_steps=30, exact_block_threshold=64)
    sums = []
    for defer in (False, True, True):
        with pkg.Engine(m, opts) as eng:
            eng.thermo_configure([2.0, 10.0], pkg.linspace(-3.0, 5.0, 17))
            eng.spectra_defer(defer)
            for nu in range(2, 7):
                for nd in range(2, 7):
                    info = eng.sector_prepare(nu, nd)
                    blocks = [(k % 3, k // 3) for k in range(9)]
                    eng.blocks_ftlm_batched(blocks)
                    for b in blocks:
                        eng.thermo_accumulate_block(*b)
            sums.append(eng.thermo_read())
            eng.spectra_defer(False)
            assert all(info.block_dims)
    for s in sums[1:]:
        for a, b in zip(s, sums[0]):
            assert np.array_equal(a, b)
