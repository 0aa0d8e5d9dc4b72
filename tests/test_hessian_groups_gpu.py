"""GPU: the Hessian at the numbers of rank x wave slots where its Gram columns
(two per slot and one) are split into groups of 48 differently: the last single
Gram, the first split, slots that fill whole groups, several ranks over the
groups' edges.  Against the FP64 oracle, tolerance as in test_hessian_gpu.py;
no block may be left at zero."""
import numpy as np
import pytest

from rootpwa_gb300 import synth
import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_neg,n_pos,rank", [(0, 47, 1), (0, 48, 1), (5, 44, 1), (0, 48, 2), (4, 20, 4), (3, 27, 4),
                                              (0, 48, 3), (10, 35, 3)])
def test_groups(n_neg, n_pos, rank, monkeypatch):
    monkeypatch.setitem(synth.WORKLOADS, "groups", dict(n_neg=n_neg, n_pos=n_pos, rank=rank, n_data=1501, n_mc=4000,
                                                        mixing=0))
    w = synth.make_workload("groups", seed=n_pos + rank)
    norm, acc, gn, ga = helpers.integral_pairs(w)
    H0 = helpers.build_oracle(w, norm, acc).Hessian(w["par"])
    H1 = helpers.build_gpu(w, gn, ga).Hessian(w["par"])
    assert np.max(np.abs(H1 - H0)) / np.max(np.abs(H0)) < 2e-5
    # and relative to the two parameters' own curvatures
    d = np.sqrt(np.abs(np.diag(H0)))
    assert np.max(np.abs(H1 - H0) / np.outer(d, d)) < 1e-3
    assert np.array_equal(H1, H1.T)
    assert not np.any((H1 == 0) & (np.abs(H0) > 1e-9 * np.max(np.abs(H0))))
