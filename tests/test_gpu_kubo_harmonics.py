"""The conductivity from the moment matrix's diagonal and antidiagonal sums:
one and two moments, fewer nodes than harmonics, odd node counts with the
middle node at the Fermi energy, nodes up to the band edge, a strided moment
matrix without symmetry, and node counts that leave a block ragged."""
import math

import numpy as np
import pytest

import kpm_gb300 as kg
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("beta", [math.inf, 10.0])
@pytest.mark.parametrize("NC,quad_N,cutoff", [
    (1, 8, 1e-3), (2, 33, 1e-3), (3, 1, 0.0), (31, 7, 0.0), (64, 511, 1e-3), (130, 1040, 0.3),
    (257, 96, 1e-3)])
def test_matches_oracle(NC, quad_N, cutoff, beta):
    rng = np.random.default_rng(NC)
    n = np.arange(NC + 5)
    env = np.exp(-(n[:, None] + n[None, :]) / (NC / 3 + 1))
    mu = (rng.standard_normal(env.shape) + 1j * rng.standard_normal(env.shape)) * env
    kw = dict(b=0.25, NH=100, area=50.0, NC=NC, quad_N=quad_N, edge_cutoff=cutoff, beta=beta)
    Ef = np.array([-1.9, 0.25, 0.3, 1.7])
    got = kg.kubo_bastin_cond(mu, 2.0, Ef, **kw)
    ref = np.array([ko.kubo_bastin_cond(mu, 2.0, e, **kw) for e in Ef])
    # the node sums add (2 NC)^2 terms of FP64, with weights 1/s^3 up to the
    # cut-off: the tolerance of the reconstruction tests
    assert np.abs(got - ref).max() <= 1e-11 * max(np.abs(ref).max(), 1e-3)
