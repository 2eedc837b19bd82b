"""Wide stencil sweeps of the split-spin H*V (k_hv_stn) at the sizes where
their tiling can go wrong, against the oracle CSR (apply_hamiltonian,
main.cpp:833-845): blocks smaller than one work unit, segments of 1 to a few
hundred rows, classes with fewer segments than a warp takes, sectors with one
particle of a spin, hops to inactive orbits, 33 sites (64-bit words), every
width and every variant.

Bound per row: a row adds h hops of rounded coefficients, and the diagonal;
each complex multiply-add rounds at most 4 times per component, the inputs
and coefficients once, so |y - Hx| <= 4 (h + 4) u (|H| |x|), u = 2^-53 or
2^-24 (|z| taken as |re| + |im|).
"""
import numpy as np
import pytest

import pyoracle as O

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

pytestmark = pytest.mark.gpu

# lx, ly, N_up, N_down, mx, my
BLOCKS = [(2, 2, 2, 2, 1, 0), (3, 2, 3, 3, 0, 0), (6, 1, 3, 2, 2, 0), (4, 2, 4, 4, 0, 0), (4, 2, 1, 7, 3, 1),
          (3, 3, 4, 2, 1, 2), (4, 4, 2, 3, 0, 2), (4, 4, 1, 8, 2, 0), (6, 3, 2, 2, 3, 0), (11, 3, 1, 2, 5, 1)]


def model(lx, ly):
    return pkg.Model(lx=lx, ly=ly, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)


def cabs(z):
    return np.abs(z.real) + np.abs(z.imag)


@pytest.mark.parametrize("block", BLOCKS, ids=lambda b: "%dx%d_%d_%d_k%d%d" % b)
@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED], ids=["fp64", "mixed"])
def test_wide_sweeps_match_the_oracle(monkeypatch, block, prec):
    lx, ly, nu, nd, mx, my = block
    m = model(lx, ly)
    csr = O.block_csr(O.Model(**m.__dict__), nu, nd, mx, my)
    rng = np.random.default_rng(3)
    monkeypatch.setenv("FTLM_HV_MODE", "split")
    monkeypatch.setenv("FTLM_STN_ROWS", "0")  # the wide kernel at every width
    u = 2.0 ** -53 if prec == E.PREC_FP64 else 2.0 ** -24
    hops = np.diff(csr.row_ptr)
    mag = cabs(csr.val)
    for nvec in (1, 3, 7, 16, 33, 128):
        x = rng.standard_normal((csr.dim, nvec)) + 1j * rng.standard_normal((csr.dim, nvec))
        if prec == E.PREC_MIXED:
            x = x.astype(np.complex64).astype(np.complex128)
        want = np.stack([csr.apply(np.ascontiguousarray(x[:, v])) for v in range(nvec)], 1)
        size = np.abs(csr.diag)[:, None] * cabs(x)
        np.add.at(size, np.repeat(np.arange(csr.dim), hops), mag[:, None] * cabs(x[csr.col]))
        bound = 4.0 * (hops[:, None] + 4) * u * size
        for var in range(5):
            monkeypatch.setenv("FTLM_HV_VARIANT", str(var))
            with pkg.Engine(m, pkg.RunOpts(precision=prec)) as eng:
                eng.sector_prepare(nu, nd)
                eng.profile_reset()
                y = eng.block_apply(mx, my, x)
                assert eng.profile()["hv_source"] == 2
            assert np.all(cabs(y - want) <= bound), (nvec, var, (cabs(y - want) / np.maximum(bound, 1e-300)).max())


@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED], ids=["fp64", "mixed"])
def test_lanczos_coefficients_do_not_depend_on_the_variant(monkeypatch, prec):
    """The dot products are exact sums of per-unit terms: alpha and beta are
    the same bits for every CTA shape and for rows taken grid-stride."""
    m = model(4, 4)
    opts = pkg.RunOpts(samples=24, lanczos_steps=8, exact_block_threshold=0, precision=prec,
                       start_vector=E.START_PHILOX_PHASE)
    monkeypatch.setenv("FTLM_HV_MODE", "split")
    got = []
    for var, rows in [(v, "") for v in range(5)] + [(2, "stride")]:
        monkeypatch.setenv("FTLM_HV_VARIANT", str(var))
        monkeypatch.setenv("FTLM_SEG_ROWS", rows)
        with pkg.Engine(m, opts) as eng:
            eng.sector_prepare(3, 2)
            got.append(eng.block_lanczos(1, 2))
    for a, b, s in got[1:]:
        assert np.array_equal(a, got[0][0]) and np.array_equal(b, got[0][1]) and np.array_equal(s, got[0][2])


@pytest.mark.parametrize("prec,tol", [(E.PREC_FP64, 1e-11), (E.PREC_MIXED, 2e-4)], ids=["fp64", "mixed"])
def test_vectors_per_sweep_do_not_change_the_coefficients(monkeypatch, prec, tol):
    """The row order of the sweeps depends on their width, and the last sweep
    of a block is narrower than the others: 21 vectors in one sweep, in 16 + 5,
    in 7 + 7 + 7 and singly give the same alpha and beta up to the rounding of
    the update (u times the amplification of 6 steps, below 1e5 u here)."""
    monkeypatch.setenv("FTLM_HV_MODE", "split")
    monkeypatch.setenv("FTLM_HV_VARIANT", "1")
    got = {}
    for batch in (21, 16, 7, 1):
        opts = pkg.RunOpts(samples=21, lanczos_steps=6, exact_block_threshold=0, precision=prec,
                           batch_vectors=batch, start_vector=E.START_PHILOX_PHASE)
        with pkg.Engine(model(4, 4), opts) as eng:
            eng.sector_prepare(3, 2)
            got[batch] = eng.block_lanczos(1, 2)
    a, b, s = got[21]
    for batch in (16, 7, 1):
        assert np.array_equal(got[batch][2], s)
        assert np.abs(got[batch][0] - a).max() <= tol * np.abs(a).max(), batch
        assert np.abs(got[batch][1] - b).max() <= tol * np.abs(b).max(), batch


@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED], ids=["fp64", "mixed"])
def test_host_vectors_of_every_size_are_the_same_vectors(monkeypatch, prec):
    """Host vectors are converted on the host (few elements), on the device, and
    there in several chunks (more than 2^24 elements: 4x4 (5,5), 1.19 M rows, 15
    vectors). A vector's result does not depend on how it came: the same bits
    alone and among others."""
    monkeypatch.setenv("FTLM_HV_VARIANT", "1")
    for (nu, nd), widths in {((2, 3)): (3, 16), ((3, 4)): (3, 7), ((5, 5)): (15,)}.items():
        with pkg.Engine(model(4, 4), pkg.RunOpts(precision=prec)) as eng:
            dim = int(eng.sector_prepare(nu, nd).block_dims[0])
            for nvec in widths:
                g = np.random.default_rng(nvec)
                x = g.standard_normal((dim, nvec)) + 1j * g.standard_normal((dim, nvec))
                y = eng.block_apply(0, 0, x)
                for v in {0, nvec - 1}:
                    alone = eng.block_apply(0, 0, np.ascontiguousarray(x[:, v:v + 1]))[:, 0]
                    if dim >= 1 << 15:  # the same operator at every width
                        assert np.array_equal(alone, y[:, v]), (nu, nd, nvec, v)
                    else:
                        tol = 1e-13 if prec == E.PREC_FP64 else 2e-6
                        assert np.abs(alone - y[:, v]).max() <= tol * np.abs(y).max(), (nu, nd, nvec, v)
