"""kpmgb_kpm1d_noalloc close to what its static scratch holds, where only one
launch's columns of block sums fit beside the two slots."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NH,NR", [(2005, 1000), (6700, 300), (303, 6600)])
def test_many_columns(built_lib, NH, NR):
    import torch
    import kpm_gb300 as kg
    from kpm_gb300 import _native

    assert 0.95 * 2 ** 26 < 2 * NH * NR * 16 < 0.97 * 2 ** 26
    lib = _native.load()
    rng = np.random.default_rng(NR)
    off = rng.uniform(0.1, 0.4, NH - 1)
    H = sp.diags([off, rng.uniform(-0.1, 0.1, NH), off], [-1, 0, 1], format="csr").astype(complex)
    NC = 10
    psi = rng.standard_normal((NH, NR)) + 1j * rng.standard_normal((NH, NR))
    dev = torch.device("cuda")
    rowptr = torch.from_numpy(H.indptr.astype(np.int32)).to(dev)
    col = torch.from_numpy(H.indices.astype(np.int32)).to(dev)
    val = torch.from_numpy(H.data).to(dev)
    psi_t = torch.from_numpy(np.ascontiguousarray(psi.T)).to(dev)
    mu_t = torch.full((NC, NR), float("nan"), dtype=torch.complex128, device=dev)
    torch.cuda.synchronize()
    _native.check(lib.kpmgb_kpm1d_noalloc(
        NH, C.c_void_p(rowptr.data_ptr()), C.c_void_p(col.data_ptr()), C.c_void_p(val.data_ptr()),
        NC, NR, C.c_void_p(psi_t.data_ptr()), C.c_void_p(mu_t.data_ptr()), C.c_void_p(0)))
    torch.cuda.synchronize()
    ref = kg.kpm_1d(H.tocsc(), NC, NR, psi_in=psi, avg_output=False)
    assert relerr(mu_t.cpu().numpy().T, ref) < 1e-12
