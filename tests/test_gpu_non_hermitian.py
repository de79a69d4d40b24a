"""Doubling moments of operators that are not Hermitian: <T_{n-1} psi|T_n psi>
is complex, and the kernels chosen automatically keep its imaginary part at
every number of columns -- against the oracle's complex dots."""
import numpy as np
import pytest
import scipy.sparse as sp

from conftest import relerr
import kpm_gb300 as kg
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def _band(n, W, complex_v, rng):
    """A band with W entries in the longest row and a sizeable anti-Hermitian part."""
    H = sp.diags(rng.uniform(-0.3, 0.3, n)).astype(complex)
    for d in range(1, W // 2 + 1):
        for side in (d, -d):
            v = rng.uniform(0.1, 1.0, n - d)
            H = H + sp.diags(v + 1j * rng.uniform(-1, 1, n - d) if complex_v else v + 0j, side)
    H = H.tocsc()
    return (H / (1.5 * abs(H).sum(axis=1).max())).tocsc()


# 24000 rows: a launch per step; 3000: inside the range of a cluster per column
@pytest.mark.parametrize("n", [3000, 24000])
@pytest.mark.parametrize("W,complex_v,columns", [
    (5, False, [1, 2, 5, 8, 12, 40, 64, 65, 128]),
    (7, False, [3, 8, 50, 64, 100]),
    (5, True, [2, 3, 8, 12, 32, 33, 48]),
    (11, True, [2, 7, 16, 40, 128]),
])
def test_doubling_moments(n, W, complex_v, columns):
    rng = np.random.default_rng(W)
    H = _band(n, W, complex_v, rng)
    assert np.diff(H.tocsr().indptr).max() == W
    psi = ko.random_phase_vectors(rng, n, max(columns))
    ref = ko.kpm_1d_doubling(H, 12, psi)
    odd = ref[:, 1::2]
    assert np.abs(odd.imag).max() > 1e-4 * np.abs(odd.real).max()
    op = kg.GB300Operator(H)
    for NR in columns:
        got = kg.kpm_1d(op, 12, NR, psi_in=psi[:, :NR], avg_output=False, precision="ff")
        # 48-bit values: 2^-48 a step and product, growing with the square of 6 steps
        assert relerr(got, ref[:NR]) < 1e-11, NR


def _with_parts(A, split):
    """A with some entries (row, column) stored in two parts."""
    A = A.tocoo()
    row, col, val = A.row.tolist(), A.col.tolist(), A.data.copy()
    for (i, j), f in split.items():
        k = next(k for k in range(len(row)) if row[k] == i and col[k] == j)
        row.append(i)
        col.append(j)
        val = np.append(val, f * val[k])
        val[k] *= 1 - f
    order = np.lexsort((row, col))
    row, col, val = np.array(row)[order], np.array(col)[order], val[order]
    indptr = np.searchsorted(col, np.arange(A.shape[1] + 1))
    return sp.csc_matrix((val, row, indptr), shape=A.shape)


@pytest.mark.parametrize("case", ["one-sided", "parts", "unequal parts"])
def test_decided_by_sums(case):
    """An entry without its mirror, and entries stored in several parts: what
    counts are the sums they stand for."""
    rng = np.random.default_rng(3)
    n, NR = 30000, 4
    A = _band(n, 5, False, rng)
    A = ((A + A.T.conj()) / 2).tocsc()
    if case == "one-sided":
        A = A.tolil()
        A[17, 900] = 0.2
        A = A.tocsc()
    else:
        B = _with_parts(A, {(40, 41): 0.25, (41, 40): 0.75, (50, 50): 0.5, (70, 68): 0.5})
        assert B.nnz == A.nnz + 4
        if case == "unequal parts":
            B.data[B.indptr[41]:B.indptr[42]] *= 1.5
        A = B
    psi = ko.random_phase_vectors(rng, n, NR)
    got = kg.kpm_1d(A, 8, NR, psi_in=psi, avg_output=False, precision="ff")
    assert relerr(got, ko.kpm_1d_doubling(A, 8, psi)) < 1e-11
