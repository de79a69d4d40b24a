"""The double-precision contraction keeps the accuracy of FP64 sums for
vectors of any dynamic range: every moment is compared by itself, relative to
the sum of its terms' moduli, with the exact sum."""
import math

import numpy as np
import pytest
import scipy.sparse as sp

import kpm_gb300 as kg

pytestmark = pytest.mark.gpu

NC = 8


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    return built_lib


def _moment(pl, pr, **kw):
    """mu[0, 0] = sum conj(pl) pr: H = 0 and unit currents."""
    NH = pl.shape[0]
    zero = sp.csc_matrix((np.zeros(NH), (np.arange(NH), np.arange(NH))), shape=(NH, NH))
    one = sp.identity(NH, format="csc")
    return kg.kpm_2d(zero, one, one, NC, 1, NH, psi_in_l=pl[:, None], psi_in_r=pr[:, None],
                     **kw)[0, 0]


def _parts(a, b):
    re = np.concatenate([a.real * b.real, a.imag * b.imag])
    im = np.concatenate([a.real * b.imag, -a.imag * b.real])
    return re, im


def _check(pl, pr, precision="fp64"):
    got = _moment(pl, pr, precision=precision)
    # float-float vectors hold every part to 2^-48 of itself
    held = {"fp64": 0.0, "ff": 2.0 ** -46}[precision]
    # products in 80-bit numbers: their rounding is far below the bound
    x, y = pl.astype(np.clongdouble), pr.astype(np.clongdouble)
    for value, terms in zip((got.real, got.imag), _parts(x, y)):
        exact = math.fsum(map(float, terms))
        # n FP64 additions and the final sums, each 2^-53 of at most the sum of moduli
        bound = ((2 * len(pl) + 64) * 2.0 ** -53 + held) * float(np.abs(terms).sum())
        assert abs(value - exact) <= bound + 1e-300, (value, exact)


@pytest.mark.parametrize("precision", ["fp64", "ff"])
@pytest.mark.parametrize("width,gap", [(150.0, 1800), (150.0, 2300), (110.0, 1900), (400.0, 1000)])
def test_packets_far_apart(width, gap, precision):
    """Two packets whose overlap is far below the product of their norms."""
    n = 3000
    i = np.arange(n)
    mid = n / 2
    pl = np.exp(-(i - mid + gap / 2) ** 2 / (2 * width ** 2)) * np.exp(0.1j * i)
    pr = np.exp(-(i - mid - gap / 2) ** 2 / (2 * width ** 2)) * np.exp(0.1j * i + 0.3j)
    _check(pl, pr, precision)


@pytest.mark.parametrize("side,precision", [("left", "fp64"), ("right", "fp64"), ("left", "ff")])
@pytest.mark.parametrize("small", [1e-6, 1e-12, 1e-20, 1e-40])
def test_small_imaginary_part(small, side, precision):
    """A real vector against one with a small imaginary part.  (The right one
    passes through the currents' steps, which hold float-float parts relative
    to the larger of the two; 1e-40 is below the floats' range.)"""
    if precision == "ff" and small < 1e-30:
        return
    rng = np.random.default_rng(1)
    n = 20011
    a = rng.uniform(0.5, 1.5, n) + 0j
    b = rng.uniform(0.5, 1.5, n) + 1j * small * rng.uniform(0.5, 1.5, n)
    _check(*((a, b) if side == "right" else (b, a)), precision)


@pytest.mark.parametrize("span,precision", [(4, "fp64"), (9, "fp64"), (40, "fp64"), (200, "fp64"),
                                            (4, "ff"), (40, "ff")])
def test_graded_vectors(span, precision):
    """Entries falling over 2^-span of the largest, in opposite directions."""
    n = 9001
    k = np.arange(n) / n
    phase = np.exp(2j * np.pi * 0.01 * np.arange(n))
    _check(np.exp2(-span * k) * phase, np.exp2(-span * (1 - k)) * phase, precision)


@pytest.mark.parametrize("precision", ["fp64", "ff"])
@pytest.mark.parametrize("spike", [1.0, 8.0, 31.0, 33.0, 500.0, 1e5])
def test_spiked_vectors(spike, precision):
    """A single large entry on either side of the bound on peaks."""
    rng = np.random.default_rng(7)
    n = 8200
    pl, pr = (rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))) / 2
    pl[5] *= spike
    pr[n - 5] *= spike
    _check(pl, pr, precision)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite(bad):
    rng = np.random.default_rng(2)
    n = 5000
    pl, pr = rng.standard_normal((2, n)) + 0j
    pr[1234] = bad
    assert not np.isfinite(_moment(pl, pr))


def test_zero_vectors():
    n = 4097
    assert _moment(np.zeros(n, complex), np.ones(n, complex)) == 0
    half = (np.arange(n) % 2).astype(complex)
    assert _moment(half, np.ones(n, complex)) == n // 2
    assert _moment(half, 1 - half) == 0


def _halves(rng, n, left, right):
    """Gaussian vectors whose halves have the given sizes."""
    h = n // 2
    out = []
    for sizes in (left, right):
        v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        v[:h] *= sizes[0]
        v[h:] *= sizes[1]
        out.append(v)
    return out


@pytest.mark.parametrize("n", [5000, 16384, 41003])
@pytest.mark.parametrize("left,right", [((1, 1), (1, 1)), ((1, 0), (0.04, 1)), ((1, 0), (0, 1)),
                                        ((1, 1e-9), (1e-9, 1)), ((1, 0.1), (0, 1))]
                         + [((1, 2.0 ** -k), (2.0 ** -k, 1)) for k in (3, 5, 6, 7, 8, 9, 12)])
def test_halves_of_different_size(n, left, right):
    """Terms far below the product of the maxima: the sum is as near to the
    exact one as FP64 sums over runs of 1024 products and more are."""
    rng = np.random.default_rng(n)
    pl, pr = _halves(rng, n, left, right)
    got = _moment(pl, pr)
    x, y = pl.astype(np.clongdouble), pr.astype(np.clongdouble)
    for value, terms in zip((got.real, got.imag), _parts(x, y)):
        exact = math.fsum(map(float, terms))
        # root mean square 0.42 2^-54 sqrt(run) per product, twelve of them (the
        # figure is measured to within 2), and the rounding of the sums' total
        size = float(np.sqrt((terms.astype(float) ** 2).sum()))
        bound = 12 * 0.42 * 2.0 ** -54 * math.sqrt(1024) * size + 16 * 2.0 ** -53 * abs(exact)
        assert abs(value - exact) <= bound, (value, exact)
