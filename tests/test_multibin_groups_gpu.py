"""GPU test of the batched FdF at the edges of its thread layout: wave counts
around the four waves of a warp and the 32 of the first wave set (1 to 64),
groups with one start, an odd last start and a full second group, and bins that
end inside a tile and inside a folding window of eight tiles.

Every problem against its bin's own likelihood (itself checked against the FP64
oracle): 1e-5 normwise in the gradient, and in f 1e-6 relative plus, as f is a
small difference of large sums here, 2^-21 per event: an event's L carries a
relative rounding error of about 2^-22 in either path, which is the absolute
error of its ln L however far the sums cancel."""
import numpy as np
import pytest

import rootpwa_gb300 as R
import helpers

pytestmark = pytest.mark.gpu


def _integral(names, diag, n):
    I = R.ampIntegralMatrix()
    I.setWaveNames(names)
    I.setMatrix(np.diag(diag).astype(np.complex128) * n)
    I.setNmbEvents(n)
    return I


def _bin(names, n, rng):
    scale = np.exp(rng.uniform(-1, 1, len(names)))
    L = R.pwaLikelihood()
    L.init(names, [1] * len(names), None, 1, 0.0)
    L.addNormIntegral(_integral(names, 2 * scale ** 2, 1000))
    L.addAccIntegral(_integral(names, scale ** 2, 600))
    for k, name in enumerate(names):
        z = rng.standard_normal((2, n)) * scale[k]
        L.addAmplitude(name, (z[0] + 1j * z[1]).astype(np.complex64))
    L.setAutotune(False)
    L.finishInit()
    return L


@pytest.mark.parametrize("W", [1, 3, 4, 5, 31, 32, 33, 36, 37, 50, 63, 64])
@pytest.mark.parametrize("group", [32, 8])
def test_wave_counts_and_ragged_groups(W, group):
    rng = np.random.default_rng(100 * W + group)
    names = ["p%02d" % i for i in range(W)]
    bins = [(_bin(names, n, rng), n, s) for n, s in ((1, 1), (129, 33), (1025, 64), (2305, 7))]
    M = R.pwaMultibin()
    M.setOptions(startGroup=group)
    for L, _, s in bins:
        M.addBin(L, s)
    x = rng.standard_normal((M.nmbProblems(), M.nmbPars()))
    f, g = M.FdF(x)
    q = 0
    for L, n, s in bins:
        for k in range(s):
            if k in (0, 1, 6, 31, 32, s - 1):
                f1, g1 = L.FdF(x[q + k])
                assert abs(f[q + k] - f1) < 1e-6 * abs(f1) + n * 2.0 ** -21, (q, k)
                assert helpers.normwise(g[q + k], g1) < 1e-5, (q, k)
        q += s
    # the same bits again, and with a problem's neighbours changed
    x2 = x.copy()
    x2[1::2] *= 0.5
    f2, g2 = M.FdF(x2)
    assert np.array_equal(f[::2], f2[::2]) and np.array_equal(g[::2], g2[::2])
