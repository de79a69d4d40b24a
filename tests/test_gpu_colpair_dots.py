"""Moments of complex operators on column pairs: every lane count, odd column
counts (half a pair), rows of 5..12 entries, and lanes that fold their sums."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import relerr
import kpm_gb300 as kg
from kpm_gb300 import models
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def _band(n, W, rng):
    """Hermitian band with W entries in the longest row (W odd)."""
    H = sp.diags(rng.uniform(-0.3, 0.3, n)).astype(complex).tocsr()
    for d in range(1, W // 2 + 1):
        v = rng.standard_normal(n - d) + 1j * rng.standard_normal(n - d)
        H = H + sp.diags(v, d) + sp.diags(v.conj(), -d)
    return (H / (1.02 * abs(H).sum(axis=1).max())).tocsc()


@pytest.mark.parametrize("NR", [2, 3, 4, 5, 8, 9, 13, 16, 27, 31, 32])
@pytest.mark.parametrize("lr", [False, True])
def test_haldane(NR, lr):
    rng = np.random.default_rng(NR)
    H, _, _, _ = models.haldane(130, 95)
    H = (H / 4.5).tocsc()
    NH = H.shape[0]
    pr = ko.random_phase_vectors(rng, NH, NR)
    if lr:
        pl = ko.random_phase_vectors(rng, NH, NR)
        got = kg.kpm_1d(H, 31, NR, psi_in_l=pl, psi_in_r=pr, avg_output=False, precision="ff")
        assert np.abs(got - ko.kpm_1d_lr(H, 31, pl, pr)).max() < 1e-9
    else:
        got = kg.kpm_1d(H, 32, NR, psi_in=pr, avg_output=False, precision="ff")
        assert relerr(got, ko.kpm_1d_doubling(H, 32, pr)) < 1e-9


@pytest.mark.parametrize("W", [5, 7, 9, 11])
@pytest.mark.parametrize("n", [25001, 90000])
def test_bands(W, n):
    rng = np.random.default_rng(W)
    H = _band(n, W, rng)
    psi = ko.random_phase_vectors(rng, n, 6)
    got = kg.kpm_1d(H, 24, 6, psi_in=psi, avg_output=False, precision="ff")
    assert relerr(got, ko.kpm_1d_doubling(H, 24, psi)) < 1e-9
