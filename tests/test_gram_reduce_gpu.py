"""GPU: the sum of the tensor-core Gram's partials at the wave counts where its
two block shapes meet (48/49 waves for few events, 84/85 for many), at one wave
and at the widest set, against a complex128 product of the same amplitudes.

Tolerance relative to sqrt(I_ii I_jj): 2e-6, the bound that the three-product
TF32 path has in the integral tests (FP32 accumulation per CTA)."""
import numpy as np
import pytest

import rootpwa_gb300 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 2, 7, 8, 9, 48, 49, 84, 85, 86, 128])
@pytest.mark.parametrize("n", [1000, 4096, 40_002])
def test_widths(W, n):
    rng = np.random.default_rng(W * n)
    A = (rng.standard_normal((W, n)) + 1j * rng.standard_normal((W, n))).astype(np.complex64)
    I = R.ampIntegralMatrix()
    I.integrate(["w%d" % i for i in range(W)], A, precision="tf32x3")
    m = I.matrix()
    X = A.astype(np.complex128)
    ref = X @ X.conj().T
    d = np.sqrt(np.real(np.diag(ref)))
    assert np.max(np.abs(m - ref) / np.outer(d, d)) < 2e-6
    assert np.array_equal(m, m.conj().T) and np.all(np.imag(np.diag(m)) == 0)
