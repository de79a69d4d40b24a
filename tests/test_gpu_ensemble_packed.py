"""Ensembles of real float-float members on the packed step: members of one
row, one block, several blocks and ragged remainders, every lane count, a last
batch of one column, rows of 5..8 entries, and the capped held sums."""
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


def _band(n, W, rng):
    """Real symmetric band with up to W entries per row."""
    H = sp.diags(rng.uniform(-1, 1, n)).tocsr()
    for d in (1, 3, 4)[:(W - 1) // 2]:
        if d < n:
            v = rng.uniform(0.2, 1, n - d)
            H = H + sp.diags(v, d) + sp.diags(v, -d)
    if W % 2 == 0 and n > 20:       # pairs (i, i + n/2): one more entry per row
        h = n // 2
        v = np.zeros(n - h)
        v[:h] = rng.uniform(0.2, 1, h)
        H = H + sp.diags(v, h) + sp.diags(v, -h)
    return (H / (1.02 * abs(H).sum(axis=1).max())).astype(complex).tocsc()


def _check(sizes, W, NC, NR, seed):
    rng = np.random.default_rng(seed)
    Hs = [_band(n, W, rng) for n in sizes]
    psis = [ko.random_phase_vectors(rng, n, NR) for n in sizes]
    got = kg.kpm_1d_ensemble(Hs, NC, psis, precision="ff", avg_output=False)
    for H, psi, m in zip(Hs, psis, got):
        assert relerr(m, ko.kpm_1d_doubling(H, NC, psi)) < 1e-9


@pytest.mark.parametrize("NR", [2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 34])
def test_columns(NR):
    _check([1, 127, 128, 129, 1, 16, 700, 255, 257], 5, 22, NR, NR)


@pytest.mark.parametrize("W", [5, 6, 7, 8])
def test_widths(W):
    _check([64, 30000, 5, 41003], W, 24, 8, W)


def test_many_members():
    _check([20 + k % 7 for k in range(300)], 5, 2, 4, 1)


def test_sums_held_in_parts():
    # 2 x 16 x 16 bytes per block: NC / 2 steps of 2000 blocks exceed 32 MiB
    _check([97] * 2000, 5, 128, 16, 2)
