"""GPU: what an integral object keeps on the device between calls does not grow
with the number of weighted events."""
import numpy as np
import pytest

import rootpwa_gb300 as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nSub", [1, 2])
def test_event_weights_are_given_back(nSub):
    import torch
    n = 6_000_000
    a = torch.randn(2, n * nSub, dtype=torch.complex64, device="cuda")
    w = np.random.default_rng(1).uniform(0.5, 2.0, n)
    I = R.ampIntegralMatrix()
    kw = dict(precision="fp32", nmbSubAmps=nSub)
    I.integrate(["a", "b"], a, **kw)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    I.integrate(["a", "b"], a, weights=w, **kw)
    # 48 MB of weights and 48 or 96 MB of their inverses; 64 MiB may stay
    assert before - torch.cuda.mem_get_info()[0] <= 66 << 20
    # small ones stay, and a repeated call gives the same sums
    I.integrate(["a", "b"], a[:, :1000 * nSub].contiguous(), weights=w[:1000], **kw)
    m = I.matrix()
    I.integrate(["a", "b"], a[:, :1000 * nSub].contiguous(), weights=w[:1000], **kw)
    assert np.array_equal(m, I.matrix())
