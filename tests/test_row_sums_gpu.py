"""How the stencil sweeps add up a row: narrow sweeps four hops at a time,
sweeps of 32 chunks and more (64 FP32, 32 FP64 vectors) in one chain.

Bound. A row of 4x4 (3,4) adds some 14 to 28 hops a sweep, 4 roundings each, against 1
in a sum of growing size per four hops, so the variance of what the additions round off
falls to about a third; the rest of the error (coefficients, the stored sums of the two
sweeps) is the same and was two fifths of the chain's variance. Error relative to the
chain's: sqrt(2/5 + 3/5 / 3) = 0.77 in FP32. In FP64 the coefficients of momentum (1, 0) are
exact to begin with and the same holds with 1/2 for 2/5: 0.82. Both with 5% on top."""
import numpy as np
import pytest

import pyoracle as O

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

pytestmark = pytest.mark.gpu

MODEL = dict(lx=4, ly=4, tp=0.3, phix=0.3, phiy=0.7, u=7.0, v=0.5)


@pytest.fixture(scope="module")
def block():
    csr = O.block_csr(O.Model(**MODEL), 3, 4, 1, 0)
    g = np.random.default_rng(5)
    return csr, g.standard_normal((csr.dim, 64)) + 1j * g.standard_normal((csr.dim, 64))


def product(csr, x):
    """H x in extended precision."""
    x = x.astype(np.clongdouble)
    y = csr.diag.astype(np.longdouble)[:, None] * x
    rp, val = csr.row_ptr.astype(np.int64), csr.val.astype(np.clongdouble)
    n = np.diff(rp)
    for k in range(int(n.max())):
        r = np.nonzero(n > k)[0]
        y[r] += val[rp[r] + k][:, None] * x[csr.col[rp[r] + k]]
    return y


@pytest.mark.parametrize("precision,chain,widths,bound", [
    (E.PREC_MIXED, 64, (1, 2, 5, 8, 16, 31), 0.77 * 1.05), (E.PREC_FP64, 32, (1, 3, 4, 5, 8, 16), 0.82 * 1.05)],
    ids=["mixed", "fp64"])
def test_narrow_sweeps_round_less_than_a_chain(block, precision, chain, widths, bound, monkeypatch):
    monkeypatch.setenv("FTLM_HV_MODE", "split")
    csr, x = block
    if precision == E.PREC_MIXED:
        x = x.astype(np.complex64).astype(np.complex128)
    want = product(csr, x[:, :3])
    with pkg.Engine(pkg.Model(**MODEL), pkg.RunOpts(precision=precision)) as eng:
        eng.sector_prepare(3, 4)

        def error(width):
            y = eng.block_apply(1, 0, np.ascontiguousarray(x[:, :width]))
            k = min(3, width)
            d = y[:, :k] - want[:, :k]
            return float(np.sqrt((np.abs(d) ** 2).sum() / (np.abs(want[:, :k]) ** 2).sum()))

        at_chain = error(chain)
        for w in widths:
            assert error(w) <= bound * at_chain, w


@pytest.mark.parametrize("precision", [E.PREC_MIXED, E.PREC_FP64], ids=["mixed", "fp64"])
def test_infinities_stay_where_a_chain_has_them(block, precision, monkeypatch):
    """One infinite element: the same elements of the product are infinite, and the same
    are NaN, at the width of every kind of sum."""
    monkeypatch.setenv("FTLM_HV_MODE", "split")
    csr, x = block
    x = x[:, :64].copy()
    x[4321, :] = np.inf
    out = []
    with pkg.Engine(pkg.Model(**MODEL), pkg.RunOpts(precision=precision)) as eng:
        eng.sector_prepare(3, 4)
        for w in (64, 16, 2):
            y = eng.block_apply(1, 0, np.ascontiguousarray(x[:, :w]))[:, :2]
            out.append((np.isinf(y.real), np.isinf(y.imag), np.isnan(y.real), np.isnan(y.imag)))
    assert out[0][0].any() or out[0][2].any()
    for o in out[1:]:
        for a, b in zip(out[0], o):
            assert np.array_equal(a, b)
