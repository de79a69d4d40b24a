"""Device memory that a call takes beside its inputs."""
import numpy as np
import pytest
import scipy.sparse as sp

import kpm_gb300 as kg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("precision", ["fp64", "ff"])
def test_single_column_takes_two_slots(precision):
    import torch
    n = 1 << 23
    H = sp.diags([np.full(n - 1, 0.4), np.full(n - 1, 0.4)], [1, -1], format="csc")
    op = kg.GB300Operator(H)
    psi = torch.full((1, n), 1.0 + 0j, dtype=torch.complex128, device="cuda")
    mu = torch.empty((4, 1), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    kg.kpm_1d_device(op, 4, psi, mu, precision=precision)
    torch.cuda.synchronize()
    # two slots of 16 bytes per row, and the block sums
    assert free0 - torch.cuda.mem_get_info()[0] < 3 * n * 16
