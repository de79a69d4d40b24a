"""Moments whose per-block sums are added over many steps at once: sizes at
which the scratch buffer of block sums fills several times in one call, one
launch covers several column batches, a step has fewer entries than a warp,
and lanes fold their float-float sums into FP64 (more than 64 row tiles per
block) or never do."""
import numpy as np
import pytest

from conftest import relerr
import kpm_gb300 as kg
from kpm_gb300 import models
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu

# the tolerances of the two precisions (kpm_1d tests)
TOL = {"fp64": 1e-12, "ff": 1e-9}


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("L,NR,NC", [
    (150, 130, 66),    # two column batches, several fillings of the scratch
    (170, 1, 400),     # one column: two entries per step
    (40, 3, 2),        # only the first step
    (40, 3, 4),        # one later step
    (330, 9, 34),      # more than 64 row tiles per block
    (130, 33, 20),     # 66 entries: a ragged third chunk
    (191, 2, 64), (191, 3, 64), (191, 5, 64), (191, 8, 64),  # narrow packed rows
])
def test_doubling(L, NR, NC, prec):
    rng = np.random.default_rng(L)
    H = (models.square_anderson(L, W=2.0, rng=rng) / 5.1).tocsc()
    psi = ko.random_phase_vectors(rng, L * L, NR)
    got = kg.kpm_1d(H, NC, NR, psi_in=psi, avg_output=False, precision=prec, kernel="gather")
    assert relerr(got, ko.kpm_1d_doubling(H, NC, psi)) < TOL[prec]
    if prec == "ff":
        auto = kg.kpm_1d(H, NC, NR, psi_in=psi, avg_output=False, precision=prec)
        assert relerr(auto, got) < TOL[prec]


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("L,NR,NC", [(60, 130, 41), (150, 5, 90), (60, 2, 2), (60, 2, 3)])
def test_bra_ket(L, NR, NC, prec):
    rng = np.random.default_rng(NR)
    H, _, _, _ = models.haldane(L, L // 2)
    H = (H / 4.5).tocsc()
    pl = ko.random_phase_vectors(rng, H.shape[0], NR)
    pr = ko.random_phase_vectors(rng, H.shape[0], NR)
    got = kg.kpm_1d(H, NC, NR, psi_in_l=pl, psi_in_r=pr, avg_output=False, precision=prec,
                    kernel="gather")
    # moments of independent bra and ket are ~1/sqrt(NH); the rounding of the
    # recurrence is relative to the unit norms
    ref = ko.kpm_1d_lr(H, NC, pl, pr)
    assert np.abs(got - ref).max() < TOL[prec]


@pytest.mark.parametrize("prec", ["fp64", "ff"])
@pytest.mark.parametrize("lr", [False, True])
@pytest.mark.parametrize("L,NR,NC", [
    (6, 3, 40),      # one CTA
    (9, 1, 5),       # two CTAs, the second of fewer rows
    (33, 5, 1001),   # sixteen CTAs, odd rows
    (64, 17, 35),    # clusters that share SMs
    (40, 28, 3000),  # two launches: the slots pass through global memory
])
def test_cluster(L, NR, NC, lr, prec):
    rng = np.random.default_rng(L + NR)
    if lr:
        H, _, _, _ = models.haldane(L, max(3, L // 3))
        H = (H / 4.5).tocsc()
    else:
        H = (models.square_anderson(L, W=2.0, rng=rng) / 5.1).tocsc()
        NC += NC % 2
    NH = H.shape[0]
    pr = ko.random_phase_vectors(rng, NH, NR)
    if lr:
        pl = ko.random_phase_vectors(rng, NH, NR)
        got = kg.kpm_1d(H, NC, NR, psi_in_l=pl, psi_in_r=pr, avg_output=False, precision=prec,
                        kernel="cluster")
        assert np.abs(got - ko.kpm_1d_lr(H, NC, pl, pr)).max() < TOL[prec]
    else:
        got = kg.kpm_1d(H, NC, NR, psi_in=pr, avg_output=False, precision=prec, kernel="cluster")
        assert relerr(got, ko.kpm_1d_doubling(H, NC, pr)) < TOL[prec]
