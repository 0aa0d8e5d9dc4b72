"""CPU: a wave plan that needs several batches gives each wave the amplitude
that it has in a plan of its own, bit for bit: the kernel's arithmetic as host
code (the shim of test_isobar_host.py).  700 mass bins of a freed isobar, with
waves of other families before, between and after them, close batches at
several places."""
import numpy as np
import pytest

from isobar_cases import events, waves
from oracle import isobar_oracle as O
from test_isobar_host import _shim_amps, shim  # noqa: F401 (fixture)


def _bins(n):
    edges = np.linspace(0.28, 2.2, n + 1)
    out = []
    for lo, hi in zip(edges[:-1], edges[1:]):
        out.append((O.wave(0, -1, 0, +1, 0, 0, 0, 0, O.MASSDEP_BINNED, 0.0, 0.0, (1, 2), 0, False, bounds=(lo, hi)),
                    dict(J=0, P=-1, M=0, refl=+1, L=0, S=0, isobarJ=0, isobarL=0, massDependence="binned",
                         isobarMass=0.0, isobarWidth=0.0, isobarDaughters=(1, 2), bachelor=0, bounds=(lo, hi))))
    return out


@pytest.mark.parametrize("opts", [{}, {"bose": False}, {"formalism": "canonical"}],
                         ids=["default", "no-bose", "canonical"])
def test_several_batches(shim, opts):  # noqa: F811
    other, bins = waves(), _bins(700)
    k = len(other) // 2
    ws = other[:k] + bins[:350] + other[k:] + bins[350:] + other[:k]
    beam, fs, masses, mb = events(40, seed=6)
    got = _shim_amps(shim, ws, beam, fs, masses, mb, opts)
    for i, w in enumerate(ws):
        assert np.array_equal(got[i], _shim_amps(shim, [w], beam, fs, masses, mb, opts)[0]), i
