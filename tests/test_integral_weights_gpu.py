"""GPU: integrals with one weight per event (no bin selection), which are
inverted and summed on the device, against the FP64 oracle: sub-amplitudes, an
upper limit of events, more weights than events, in every precision; weights
that a precision cannot take and a stream that is too short are refused.
Tolerances as in test_integral_gpu.py."""
import numpy as np
import pytest

import rootpwa_gb300 as R
from oracle.oracle import OracleIntegral
from test_integral_gpu import TOL, maxrel

pytestmark = pytest.mark.gpu

NAMES = ["w%d" % k for k in range(9)]


def _draw(n, nSub, seed):
    rng = np.random.default_rng(seed)
    shape = (9, n, nSub) if nSub > 1 else (9, n)
    return rng, (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("nSub", [1, 2])
@pytest.mark.parametrize("limit,surplus", [(0, 0), (3501, 0), (3501, 700), (0, 5)])
def test_one_weight_per_event(precision, nSub, limit, surplus):
    n = 4001
    rng, A = _draw(n, nSub, 3 + nSub)
    wts = rng.uniform(0.2, 3.0, n + surplus)
    O = OracleIntegral()
    assert O.integrate(NAMES, A.astype(np.complex128), weights=wts, max_nmb_events=limit)
    I = R.ampIntegralMatrix()
    I.integrate(NAMES, A, weights=wts, maxNmbEvents=limit, precision=precision, nmbSubAmps=nSub)
    assert I.nmbEvents() == O.nmb_events()
    assert maxrel(I.matrix(), O.raw()) < TOL[precision]


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
def test_refused_weights(precision):
    n = 500
    rng, A = _draw(n, 1, 9)
    wts = rng.uniform(0.2, 3.0, n)
    with pytest.raises(Exception, match="shorter"):
        R.ampIntegralMatrix().integrate(NAMES, A, weights=wts[:-1], precision=precision)
    wts[77] = -1.0
    if precision == "tf32x3":
        with pytest.raises(Exception, match="non-negative"):
            R.ampIntegralMatrix().integrate(NAMES, A, weights=wts, precision=precision)
    else:
        O, I = OracleIntegral(), R.ampIntegralMatrix()
        assert O.integrate(NAMES, A.astype(np.complex128), weights=wts)
        I.integrate(NAMES, A, weights=wts, precision=precision)
        assert maxrel(I.matrix(), O.raw()) < TOL[precision]
