"""GPU test of the batched L-BFGS step at the edges of its two forms: vectors in
registers up to 128 parameters (64 waves of rank 1 have exactly 128), in memory
beyond, histories shorter and longer than a warp, and an odd number of problems
(the finish kernel takes two per block).

A fit's reported value and gradient norm are those of the batch evaluation at
its end point, to the last bit (both come from the same kernels); it ends
converged or at the rounding floor, below its start value."""
import numpy as np
import pytest

import rootpwa_gb300 as R
from test_multibin_groups_gpu import _bin, _integral

pytestmark = pytest.mark.gpu


def _rank2(W, n, rng):
    names = ["p%02d" % i for i in range(W)]
    L = R.pwaLikelihood()
    L.init(names, [1] * W, None, 2, 0.0)
    L.addNormIntegral(_integral(names, np.full(W, 2.0), 1000))
    L.addAccIntegral(_integral(names, np.full(W, 1.0), 600))
    for name in names:
        z = rng.standard_normal((2, n))
        L.addAmplitude(name, (z[0] + 1j * z[1]).astype(np.complex64))
    L.setAutotune(False)
    L.finishInit()
    return L


@pytest.mark.parametrize("W,rank,memory", [(1, 1, 1), (16, 1, 8), (17, 1, 3), (64, 1, 8), (33, 1, 40), (36, 2, 8)])
def test_fit_ends_where_it_says(W, rank, memory):
    rng = np.random.default_rng(10 * W + memory)
    names = ["p%02d" % i for i in range(W)]
    M = R.pwaMultibin()
    M.setOptions(startGroup=8, lbfgsMemory=memory, maxIter=400)
    for n, s in ((3000, 2), (1700, 3)):
        M.addBin(_bin(names, n, rng) if rank == 1 else _rank2(W, n, rng), s)
    P = M.nmbPars()
    assert (P <= 128) == (rank == 1)
    x0 = rng.standard_normal((M.nmbProblems(), P))
    f0, _ = M.FdF(x0)
    r = M.fit(x0)
    assert np.all(np.isin(r["status"], [2, 4, 6])), r["status"]
    assert np.all(r["f"] < f0) and np.all(r["iterations"] > 0)
    f, g = M.FdF(r["x"])
    assert np.array_equal(f, r["f"])
    assert np.max(np.abs(np.linalg.norm(g, axis=1) - r["gnorm"])) <= 1e-13 * np.max(r["gnorm"])
