"""Which launches a block_apply call makes: few elements are converted on the host,
many on the GPU, with equal results (the conversions round and order the same); near
full memory the operator is chosen by what the vectors leave; one
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


def _leave_free(bytes_free):
    """Holds device memory so that `bytes_free` are left."""
    import torch
    hold, fill = [], torch.cuda.mem_get_info()[0] - bytes_free
    while fill > 0:  # in pieces, so that no single one is refused
        n = min(fill, 8 << 30)
        hold.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
        fill -= n
    return hold


def test_little_memory_falls_back():
    """4x4 (8,8), 8 FP64 vectors, 1.33 GB an array: with 5.35 GB free the two vectors fit, but not
    the split sweeps' two arrays, maps and 2 GiB of headroom beside them: the on-the-fly
    kernel runs, and its H*V is that of the sweeps (60 hops of |x| <= 1 to FP64 rounding)."""
    import torch
    free = torch.cuda.mem_get_info()[0]
    if free < 20 << 30:
        pytest.skip("needs 20 GB of device memory")
    out = []
    for leave in (None, 5_350_000_000):
        with _engine(4, 4, E.PREC_FP64) as eng:
            dim = int(eng.sector_prepare(8, 8).block_dims[1])
            x = np.cos(np.arange(dim * 8, dtype=np.float64).reshape(dim, 8) * 0.37) + 0j
            hold = _leave_free(leave) if leave else []
            y = eng.block_apply(1, 0, x)
            out.append((y[::97].copy(), eng.profile()["hv_source"]))
            del hold
            torch.cuda.empty_cache()
    assert out[0][1] == 2 and out[1][1] == 0
    assert np.abs(out[0][0] - out[1][0]).max() <= 60 * 2.0 ** -53 * 16 * 100


def test_less_memory_than_a_conversion_chunk(monkeypatch):
    """4x4 (8,8), 8 FP32 vectors, 0.66 GB an array: with the two vectors, the block's tables
    (0.15 GB) and 0.15 GB more there is no room for the 256 MB of a conversion chunk."""
    import torch
    monkeypatch.setenv("FTLM_HV_MODE", "fly")
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB of device memory")
    out = []
    for short in (False, True):
        with _engine(4, 4, E.PREC_MIXED) as eng:
            dim = int(eng.sector_prepare(8, 8).block_dims[1])
            x = np.cos(np.arange(dim * 8, dtype=np.float64).reshape(dim, 8) * 0.37) + 0j
            hold = _leave_free(2 * dim * 8 * 8 + 300_000_000) if short else []
            out.append(eng.block_apply(1, 0, x)[::97].copy())
            del hold
            torch.cuda.empty_cache()
    assert np.array_equal(out[0], out[1])
