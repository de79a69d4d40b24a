"""Columns that run in several parts of one launch: parts of every width,
ragged last parts, and both sides of each rule that picks the width."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import relerr
import kpm_gb300 as kg
from kpm_gb300 import models
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "ff": 1e-9}


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("prec", ["ff", "fp64"])
@pytest.mark.parametrize("NR", [9, 11, 12, 13, 17, 20, 24, 25, 29, 33, 40, 41, 48, 49, 56, 57, 63,
                                64, 65, 72, 80, 97, 127, 128])
@pytest.mark.parametrize("lattice", ["square", "cubic", "haldane"])
def test_doubling(lattice, NR, prec):
    rng = np.random.default_rng(NR)
    H = {"square": lambda: models.square_anderson(150, W=2.0, rng=rng) / 5.1,
         "cubic": lambda: models.cubic_anderson(29, W=2.0, rng=rng) / 7.1,
         "haldane": lambda: models.haldane(110, 100)[0] / 4.5}[lattice]().tocsc()
    psi = ko.random_phase_vectors(rng, H.shape[0], NR)
    got = kg.kpm_1d(H, 12, NR, psi_in=psi, avg_output=False, precision=prec)
    assert relerr(got, ko.kpm_1d_doubling(H, 12, psi)) < TOL[prec]
    bra = ko.random_phase_vectors(rng, H.shape[0], NR)
    got = kg.kpm_1d(H, 9, NR, psi_in_l=bra, psi_in_r=psi, avg_output=False, precision=prec)
    assert np.abs(got - ko.kpm_1d_lr(H, 9, bra, psi)).max() < TOL[prec]


@pytest.mark.parametrize("W", [5, 6, 7, 8])
@pytest.mark.parametrize("n,NR", [(25001, 2), (25001, 3), (25001, 5), (300001, 8)])
def test_bra_ket_real_bands(W, n, NR):
    """Bra-ket moments of real bands on packed pairs: ragged rows of up to W
    entries, narrow columns, and lanes that fold their sums."""
    rng = np.random.default_rng(W + NR)
    H = sp.diags(rng.uniform(-1, 1, n)).tocsr()
    for d in (1, 3, 4, 7)[:W // 2]:
        v = rng.uniform(0.2, 1, n - d) * (rng.random(n - d) < 0.9)
        H = H + sp.diags(v, d) + sp.diags(v, -d)
    if W % 2 == 0:
        H = H - sp.diags(H.diagonal())
        H.eliminate_zeros()
    H = (H / (1.02 * abs(H).sum(axis=1).max())).astype(complex).tocsc()
    assert np.diff(H.indptr).max() == W
    ket, bra = (ko.random_phase_vectors(rng, n, NR) for _ in range(2))
    got = kg.kpm_1d(H, 9, NR, psi_in_l=bra, psi_in_r=ket, avg_output=False, precision="ff")
    assert np.abs(got - ko.kpm_1d_lr(H, 9, bra, ket)).max() < TOL["ff"]


@pytest.mark.parametrize("prec", ["ff", "fp64"])
@pytest.mark.parametrize("NR", [17, 33, 65, 100, 129])
def test_two_dimensional(NR, prec):
    """Batched steps without dots in parts."""
    rng = np.random.default_rng(NR)
    H, Jx, Jy, _ = models.haldane(14, 10)
    H = (H / 4.5).tocsc()
    psi = ko.random_phase_vectors(rng, H.shape[0], NR)
    got = kg.kpm_2d(H, Jx, Jy, 16, NR, H.shape[0], psi_in=psi, precision=prec)
    assert relerr(got, ko.kpm_2d(H, Jx, Jy, 16, psi, psi, 16, 16)) < TOL[prec]


@pytest.mark.parametrize("cells", [(9, 7), (15, 13)])   # K = 126 NR and 390 NR
@pytest.mark.parametrize("NR", [2, 4, 6, 8, 10, 14, 18, 20, 24, 30, 34, 40, 66])
def test_two_dimensional_column_pairs(NR, cells):
    """Column pairs without dots: every lane count and parts, with and without
    blocks of the left chain."""
    rng = np.random.default_rng(NR)
    H, Jx, Jy, _ = models.haldane(*cells)
    H = (H / 4.5).tocsc()
    psi = ko.random_phase_vectors(rng, H.shape[0], NR)
    ref = ko.kpm_2d(H, Jx, Jy, 20, psi, psi, 20, 20)
    for kw in (dict(), dict(arr_size=7, right_block=4)):
        got = kg.kpm_2d(H, Jx, Jy, 20, NR, H.shape[0], psi_in=psi, precision="ff",
                        contraction="split", **kw)
        assert relerr(got, ref) < TOL["ff"]
