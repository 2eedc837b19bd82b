"""Which launches a block_apply call makes: few elements are converted on the host,
many on the GPU, with equal results (the conversions round and order the same); one
vector without stencils goes to the hop list and builds nothing of the split sweeps."""
import numpy as np
import pytest

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

pytestmark = pytest.mark.gpu


def _engine(lx, ly, precision):
    model = pkg.Model(lx=lx, ly=ly, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)
    return pkg.Engine(model, pkg.RunOpts(precision=precision))


def _call(eng, x):
    n0 = eng.profile()["kernel_launches"]
    y = eng.block_apply(1, 0, x)
    return y, eng.profile()["kernel_launches"] - n0


# lattice, sector, vectors, precision, launches of a call: H*V alone, or with the conversions
@pytest.mark.parametrize("lx,ly,nu,nd,nvec,precision,launches", [
    (4, 2, 3, 3, 8, E.PREC_MIXED, 1),   # 3,136 elements
    (3, 3, 4, 4, 8, E.PREC_MIXED, 1),   # 14,112
    (3, 3, 4, 4, 24, E.PREC_MIXED, 3),  # 42,336
    (4, 2, 4, 4, 7, E.PREC_FP64, 1),    # 4,256, padded to 8
    (3, 3, 4, 4, 7, E.PREC_FP64, 3),    # 12,348
    (3, 3, 4, 4, 8, E.PREC_FP64, 1)])   # as it is
def test_conversions(lx, ly, nu, nd, nvec, precision, launches):
    with _engine(lx, ly, precision) as eng:
        dim = int(eng.sector_prepare(nu, nd).block_dims[1])
        rng = np.random.default_rng(2)
        x = rng.standard_normal((dim, nvec)) + 1j * rng.standard_normal((dim, nvec))
        eng.block_apply(1, 0, x)
        y, n = _call(eng, x)
        assert n == launches
        if precision == E.PREC_MIXED:
            assert np.array_equal(y, y.astype(np.complex64))
        width = 2 if precision == E.PREC_MIXED else 1  # one vector at a time: host conversions or none
        for v in range(0, nvec - width + 1, 5):
            one = eng.block_apply(1, 0, np.ascontiguousarray(x[:, v:v + width]))
            # another width groups a row's hops otherwise: hops + 2 roundings of the row's terms
            u = 2.0 ** -24 if precision == E.PREC_MIXED else 2.0 ** -53
            big = 60 * u * 8.0 * np.abs(x).max() * 8 * 16
            assert np.abs(one - y[:, v:v + width]).max() <= big


@pytest.mark.parametrize("precision", [E.PREC_FP64, E.PREC_MIXED])
def test_one_vector_without_stencils_builds_the_hop_list_only(precision, monkeypatch):
    """4x4 (3,4), 63,700 rows: as many launches from a new engine as with the list forced
    (the sweeps' tables of sector (4,3), flip map and order take about 30 more)."""
    monkeypatch.setenv("FTLM_SPLIT_OP", "fly")
    seen = []
    for mode in ("", "list"):
        if mode:
            monkeypatch.setenv("FTLM_HV_MODE", mode)
        with _engine(4, 4, precision) as eng:
            dim = int(eng.sector_prepare(3, 4).block_dims[1])
            x = np.random.default_rng(3).standard_normal((dim, 1)) + 0j
            y, n = _call(eng, x)
            seen.append((y, n, eng.profile()["hv_source"]))
    assert [s[2] for s in seen] == [1, 1]
    assert seen[0][1] == seen[1][1]
    assert np.array_equal(seen[0][0], seen[1][0])
