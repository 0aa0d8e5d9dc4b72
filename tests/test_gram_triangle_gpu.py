"""GPU: the triangle Gram kernel of the SIMT integrals at the edges of its
shapes -- groups of four waves, one and several blocks per matrix, several
chunks per block, wave sets beyond it -- against a complex128 product of the
same amplitudes, and the split FP32 arithmetic's range rule.

Tolerances: a sum of K products in FP64 carries at most about K 2^-53
relative to sum |a_i a_j|, in FP32 K 2^-24 per chunk (chunks of at most
K / 64 events are summed in FP64); the bounds are these with K = 64 steps."""
import numpy as np
import pytest

import rootpwa_gb300 as R

pytestmark = pytest.mark.gpu


def reference(A, w=None):
    X = A.astype(np.complex128)
    return (X if w is None else X * w) @ X.conj().T


def check(A, precision, tol, weights=None, inBin=None):
    names = ["w%d" % i for i in range(len(A))]
    I = R.ampIntegralMatrix()
    I.integrate(names, A, precision=precision, weights=weights, inBin=inBin)
    w = None
    if inBin is not None:
        w = inBin.astype(np.float64)
    if weights is not None:
        inv = 1.0 / weights
        w = inv * (len(inv) / inv.sum())
    ref = reference(A, w)
    m = I.matrix()
    d = np.sqrt(np.real(np.diag(ref)))
    d[d == 0] = 1.0
    assert np.max(np.abs(m - ref) / np.outer(d, d)) < tol
    assert np.array_equal(m, m.conj().T) and np.all(np.imag(np.diag(m)) == 0)


@pytest.mark.parametrize("precision,tol", [("fp64", 64 * 2.0 ** -53), ("fp32", 64 * 2.0 ** -24)])
@pytest.mark.parametrize("W,n", [(1, 1), (2, 15), (3, 17), (4, 63), (5, 129), (15, 4099), (16, 2048), (17, 3001),
                                 (50, 5003), (87, 4097), (88, 2000), (89, 2001), (112, 700), (113, 700), (224, 515), (300, 200)])
def test_shapes(W, n, precision, tol):
    rng = np.random.default_rng(1000 * W + n)
    A = (rng.standard_normal((W, n)) + 1j * rng.standard_normal((W, n))).astype(np.complex64)
    check(A, precision, tol)
    check(A, precision, tol, inBin=rng.random(n) < 0.999)
    check(A, precision, tol, weights=rng.uniform(0.2, 3.0, n))
    if precision == "fp64":
        check(A.astype(np.complex128) * (1 + 1e-12), precision, tol)


@pytest.mark.parametrize("scale", [1e-12, 1e12, 2.0 ** 61, 1e-30])
def test_range_of_the_split_sums(scale):
    """rows outside the range of the split FP32 sums, zero rows and tiny elements keep FP64 accuracy."""
    rng = np.random.default_rng(3)
    A = (rng.standard_normal((6, 5000)) + 1j * rng.standard_normal((6, 5000))).astype(np.complex64)
    A[1] *= np.float32(scale)
    A[2] = 0
    A[3, ::2] *= np.float32(1e-20)
    check(A, "fp64", 64 * 2.0 ** -53)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_amplitudes_stay_in_their_rows(bad):
    rng = np.random.default_rng(4)
    A = (rng.standard_normal((5, 5000)) + 1j * rng.standard_normal((5, 5000))).astype(np.complex64)
    A[3, 77] = bad
    I = R.ampIntegralMatrix()
    I.integrate(["w%d" % i for i in range(5)], A, precision="fp64")
    m = I.matrix()
    keep = [0, 1, 2, 4]
    ref = reference(A[keep])
    assert np.max(np.abs(m[np.ix_(keep, keep)] - ref)) < 64 * 2.0 ** -53 * np.max(np.abs(ref))
    assert not np.isfinite(m[3, 3].real) and not np.any(np.isfinite(np.abs(m[3])))
    if not np.isnan(bad):
        assert m[3, 3].real == np.inf
