"""GPU: every element of an FP64 integral is accurate relative to its own
terms -- events left out by the bin selection take no part, however large their
amplitudes are, and neither does what two waves have in other events.

Tolerance: with K = 8192 events no running sum covers more than 64 of them (128
FMAs per component), and at most 24 additions join the sums of 128 runs, so a
component is within 152 x 2^-53 and a complex element within 215 x 2^-53 of
sum_k |a_ik| |a_jk| over the selected events; 256 x 2^-53 is taken.  The exact
sums come from math.fsum over products of FP32 numbers, which FP64 holds
exactly."""
import math

import numpy as np
import pytest

import rootpwa_gb300 as R

pytestmark = pytest.mark.gpu

K = 8192
TOL = 256 * 2.0 ** -53


def draw(W, seed):
    rng = np.random.default_rng(seed)
    return rng, (rng.standard_normal((W, K)) + 1j * rng.standard_normal((W, K))).astype(np.complex64)


def check(A, inBin=None):
    I = R.ampIntegralMatrix()
    I.integrate(["w%d" % i for i in range(len(A))], A, precision="fp64", inBin=inBin)
    m = I.matrix()
    X = (A if inBin is None else A[:, inBin]).astype(np.complex128)
    for i in range(len(X)):
        for j in range(len(X)):
            a, b = X[i], X[j]
            re = math.fsum(np.concatenate([a.real * b.real, a.imag * b.imag]))
            im = math.fsum(np.concatenate([a.imag * b.real, -a.real * b.imag]))
            own = float(np.sum(np.abs(a) * np.abs(b)))
            assert abs(m[i, j] - complex(re, im)) <= TOL * own, (i, j)


@pytest.mark.parametrize("W", [1, 4, 9])
@pytest.mark.parametrize("shift", [0, 10, 20, 40])
def test_unselected_events_larger_than_the_selected(W, shift):
    rng, A = draw(W, 10 * shift + W)
    inBin = rng.random(K) < 0.5
    A[:, ~inBin] *= np.float32(2.0 ** shift)
    check(A, inBin)


@pytest.mark.parametrize("shift", [0, 10, 20, 30, 40])
def test_waves_large_in_different_events(shift):
    _, A = draw(6, shift)
    for w in range(6):
        A[w, w::6] *= np.float32(2.0 ** shift)
    check(A)


def test_one_event_outweighs_the_rest():
    _, A = draw(5, 1)
    A[0, 100] *= np.float32(2.0 ** 30)
    A[1, 4000] *= np.float32(2.0 ** 30)
    check(A)
