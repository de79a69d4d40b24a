"""The double-precision contraction on the tensor cores (eight digit planes):
tile remainders, several K ranges, blocked calls, and the FP64 kernel that
takes over for vectors peaked on few entries -- against the oracle; and its
rounding against exact sums."""
import math

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


def _check(L, NR, NC, precision, delta=False, **kw):
    rng = np.random.default_rng(NC)
    H, Jx, Jy, _ = models.haldane(L, L - 3)
    H = (H / 4.5).tocsc()
    NH = H.shape[0]
    if delta:
        pl, pr = np.zeros((NH, NR), complex), np.zeros((NH, NR), complex)
        pl[np.arange(NR), np.arange(NR)] = 1.0
        pr[np.arange(NR) + 7, np.arange(NR)] = 1.0
    else:
        pl = ko.random_phase_vectors(rng, NH, NR)
        pr = ko.random_phase_vectors(rng, NH, NR)
    got = kg.kpm_2d(H, Jx, Jy, NC, NR, NH, psi_in_l=pl, psi_in_r=pr, precision=precision, **kw)
    ref = ko.kpm_2d(H, Jx, Jy, NC, pl, pr, NC, 16)
    # the recurrences' tolerances; the contraction adds less than FP64 sums do
    assert relerr(got, ref) < (1e-12 if precision == "fp64" else 1e-9)


@pytest.mark.parametrize("precision", ["fp64", "ff"])
@pytest.mark.parametrize("L,NR,NC", [
    (32, 2, 64),     # nr, nl multiples of a tile
    (33, 3, 57),     # ragged rows, columns and K
    (60, 5, 131),    # two A tiles, the second of 3 rows; several K ranges
    (24, 7, 33),     # one row past a B tile
])
def test_matches_oracle(L, NR, NC, precision):
    _check(L, NR, NC, precision)


@pytest.mark.parametrize("kw", [dict(arr_size=50, right_block=33), dict(arr_size=7),
                                dict(moment_parity="ODD"), dict(mn_sym=True)])
def test_blocks_and_options(kw):
    rng = np.random.default_rng(5)
    H, Jx, Jy, _ = models.haldane(40, 31)
    H = (H / 4.5).tocsc()
    NH = H.shape[0]
    psi = ko.random_phase_vectors(rng, NH, 6)
    got = kg.kpm_2d(H, Jx, Jy, 72, 6, NH, psi_in=psi, **kw)
    full = kg.kpm_2d(H, Jx, Jy, 72, 6, NH, psi_in=psi,
                     **{k: v for k, v in kw.items() if k in ("moment_parity", "mn_sym")})
    assert relerr(got, full) < 1e-12


@pytest.mark.parametrize("precision", ["fp64", "ff"])
def test_peaked_vectors_take_the_fp64_kernel(precision):
    """Probes on single sites: moments of far-apart sites are tiny and keep
    their own relative accuracy."""
    _check(40, 3, 40, precision, delta=True)


def _exact_dot(a, b):
    """sum conj(a) b, correctly rounded (products split exactly)."""
    def prod(x, y):
        p = x * y
        c = 134217729.0
        xh = c * x - (c * x - x)
        yh = c * y - (c * y - y)
        xl, yl = x - xh, y - yh
        return [p, ((xh * yh - p) + xh * yl + xl * yh) + xl * yl]
    re = prod(a.real, b.real) + prod(a.imag, b.imag)
    im = prod(a.real, b.imag) + prod(-a.imag, b.real)
    return complex(math.fsum(np.concatenate(re)), math.fsum(np.concatenate(im)))


@pytest.mark.parametrize("NH,scale", [(3000, 1.0), (70001, 1.0), (70001, 1e-150)])
def test_rounding_against_exact_sums(NH, scale):
    """H = 0 leaves T_n psi = +-psi or 0, so every moment is one dot product."""
    rng = np.random.default_rng(NH)
    zero = sp.csc_matrix((np.zeros(NH), (np.arange(NH), np.arange(NH))), shape=(NH, NH))
    one = sp.identity(NH, format="csc")
    pl, pr = (rng.standard_normal((NH, 1)) + 1j * rng.standard_normal((NH, 1)) for _ in range(2))
    NC = 64
    got = kg.kpm_2d(zero, one, one, NC, 1, NH, psi_in_l=pl * scale, psi_in_r=pr) / scale
    want = _exact_dot(pl[:, 0] * scale, pr[:, 0]) / scale
    n = np.arange(NC)
    sign = np.where(n % 2 == 1, 0.0, np.where(n % 4 == 0, 1.0, -1.0))
    # a split's partial sums and their total are rounded once each (at most
    # 9 additions of 2^-53 of partial sums below the product of the norms)
    tol = 9 * 2.0 ** -53 * np.linalg.norm(pl) * np.linalg.norm(pr)
    assert np.abs(got - np.outer(sign, sign) * want).max() <= tol
