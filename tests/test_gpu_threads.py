"""Concurrent calls on distinct operators of different sizes from several
threads: every call succeeds with the values of the same call alone."""
import threading

import numpy as np
import pytest

import kpm_gb300 as kg
from kpm_gb300 import models
from oracle import kpm_oracle as ko

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


@pytest.mark.parametrize("precision", ["fp64", "ff"])
def test_small_operators(precision):
    # sizes that take a cluster per column with different shared memory, and
    # larger ones that take a launch per step
    jobs = []
    for L in (18, 33, 48, 64, 150):
        rng = np.random.default_rng(L)
        H = (models.square_anderson(L, W=2.0, rng=rng) / 5.1).tocsc()
        op = kg.GB300Operator(H)
        psi = ko.random_phase_vectors(rng, H.shape[0], 4)
        call = lambda op=op, psi=psi: kg.kpm_1d(op, 8, 4, psi_in=psi, avg_output=False,
                                                precision=precision)
        jobs.append((call, call()))
    failures = []

    def work(call, want):
        try:
            for _ in range(150):
                got = call()
                if not np.array_equal(got, want):
                    failures.append(float(np.abs(got - want).max()))
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]
