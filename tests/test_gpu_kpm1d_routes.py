"""kpm_1d on both sides of the rules that pick a schedule or a column shape:
calls of more columns than a launch or the device's clusters take at once,
operators that do not fit beside a cluster's slots, and 9..12 columns of
float-float rows that only the CSR kernel serves."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import relerr
import kpm_gb300 as kg
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "ff": 1e-11}


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def _band(n, W, complex_v, rng):
    H = sp.diags(rng.uniform(-0.3, 0.3, n)).astype(complex)
    step = max(1, int(n ** 0.5) // 2)
    for d in range(1, W // 2 + 1):
        k = d * step
        v = rng.uniform(0.1, 1, n - k) + (1j * rng.uniform(-1, 1, n - k) if complex_v else 0)
        H = H + sp.diags(v, k) + sp.diags(v.conj(), -k)
    return (H / (1.05 * abs(H).sum(axis=1).max())).tocsc()


def _check(H, NR, precision, rng):
    n = H.shape[0]
    psi, bra = (ko.random_phase_vectors(rng, n, NR) for _ in range(2))
    op = kg.GB300Operator(H)
    got = kg.kpm_1d(op, 10, NR, psi_in=psi, avg_output=False, precision=precision)
    assert relerr(got, ko.kpm_1d_doubling(H, 10, psi)) < TOL[precision]
    got = kg.kpm_1d(op, 7, NR, psi_in_l=bra, psi_in_r=psi, avg_output=False, precision=precision)
    assert np.abs(got - ko.kpm_1d_lr(H, 7, bra, psi)).max() < TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "ff"])
@pytest.mark.parametrize("complex_v", [False, True])
@pytest.mark.parametrize("n,W,NR", [
    (300, 19, 129), (1024, 5, 400), (2048, 7, 129), (2048, 19, 200), (2900, 15, 153),
    (4096, 9, 129), (9001, 19, 7), (16384, 5, 6), (20000, 3, 12),
])
def test_schedules(n, W, NR, complex_v, precision):
    rng = np.random.default_rng(n + W)
    _check(_band(n, W, complex_v, rng), NR, precision, rng)


@pytest.mark.parametrize("n", [39999, 40000, 40013])
@pytest.mark.parametrize("W,complex_v", [(3, False), (9, False), (15, True), (19, True)])
@pytest.mark.parametrize("NR", [9, 11, 12])
def test_nine_to_twelve_columns(n, W, complex_v, NR):
    rng = np.random.default_rng(NR)
    _check(_band(n, W, complex_v, rng), NR, "ff", rng)
