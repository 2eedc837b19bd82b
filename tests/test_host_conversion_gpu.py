"""Which side converts the host vectors of block_apply in mixed precision, by their
number and padding: one launch (H*V) where the host does, three where the device does.
Whole calls, host against device: 2,715 rows x 14 vectors 217 / 260 us, 14,520 x 1 153 / 131,
14,520 x 2 182 / 211, 14,520 x 3 283 / 314, 14,520 x 5 463 / 380."""
import numpy as np
import pytest

import ftlm_extended_hubbard_development_b200 as pkg
from ftlm_extended_hubbard_development_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nd,nvec,launches", [(2, 8, 14, 1), (5, 3, 1, 3), (5, 3, 2, 1), (5, 3, 3, 1), (5, 3, 5, 3)])
def test_side_of_the_conversion(nu, nd, nvec, launches, monkeypatch):
    monkeypatch.setenv("FTLM_HV_MODE", "fly")
    monkeypatch.setenv("FTLM_HV_VARIANT", "1")
    model = pkg.Model(lx=4, ly=3, tp=0.2, phix=0.3, phiy=0.7, u=7.0, v=1.5)
    with pkg.Engine(model, pkg.RunOpts(precision=E.PREC_MIXED)) as eng:
        dim = int(eng.sector_prepare(nu, nd).block_dims[1])
        rng = np.random.default_rng(2)
        x = rng.standard_normal((dim, nvec)) + 1j * rng.standard_normal((dim, nvec))
        y = eng.block_apply(1, 0, x)
        n0 = eng.profile()["kernel_launches"]
        assert np.array_equal(eng.block_apply(1, 0, x), y)
        assert eng.profile()["kernel_launches"] - n0 == launches
        last = eng.block_apply(1, 0, np.ascontiguousarray(x[:, nvec - 1:]))  # device or host, padded otherwise
        u = 2.0 ** -24
        assert np.abs(last[:, 0] - y[:, nvec - 1]).max() <= 60 * u * 8.0 * np.abs(x).max() * 8 * 16
