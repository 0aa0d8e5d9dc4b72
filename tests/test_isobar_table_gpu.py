"""GPU: the table-driven isobar amplitude kernel at the edges of its tiles
(events per block, lanes per event) and of its table (waves that need more
than one batch), against a longer run of the same events and the FP64 oracle.
Tolerances as in test_isobar_gpu.py."""
import numpy as np
import pytest

from oracle import isobar_oracle as O
from rootpwa_gb300 import isobar as I
from isobar_cases import NAMES, SPECIES, TOL, TOL32, events, tolerances, waves

pytestmark = pytest.mark.gpu


def _amp(ws, masses, mb, names=NAMES, bose=True):
    A = I.isobarHelicityAmplitudes()
    A.setFinalState(names, masses, mb)
    A.enableBoseSymmetrization(bose)
    for _, kw in ws:
        A.addWave(**kw)
    return A


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("bose", [True, False])
def test_event_counts_at_tile_edges(dtype, bose):
    """n events give the first n columns of a longer run, bit for bit."""
    beam, fs, masses, mb = events(20011, seed=3)
    A = _amp(waves(), masses, mb, bose=bose)
    full = A.amplitudes(beam, fs, dtype=dtype)
    for n in (1, 2, 15, 16, 17, 31, 33, 63, 64, 65, 127, 129, 4864, 4865, 9729, 19457):
        got = A.amplitudes(beam[:n], fs[:, :n], dtype=dtype)
        assert np.array_equal(got, full[:, :n]), n


@pytest.mark.parametrize("names,species", [(["pi-", "pi-", "pi-"], [0, 0, 0]), (["pi-", "pi-", "pi+"], [0, 0, 1]),
                                           (["pi-", "pi+", "pi0"], [0, 1, 2])])
def test_six_two_and_one_symmetrisation_terms(names, species):
    ws = waves()
    beam, fs, masses, mb = events(700, seed=4)
    ref = O.amplitudes([w for w, _ in ws], beam, fs, masses, mb, species)
    # relative to the wave's unsymmetrised amplitude: an odd-spin isobar of
    # two identical pions vanishes in the symmetrised sum
    one = O.amplitudes([w for w, _ in ws], beam, fs, masses, mb, species, bose=False)
    scale = np.abs(one).max(axis=1)
    scale[scale == 0] = 1.0
    A = _amp(ws, masses, mb, names)
    for dtype, tol in (("complex128", TOL), ("complex64", TOL32)):
        err = np.abs(A.amplitudes(beam, fs, dtype=dtype) - ref).max(axis=1) / scale
        assert np.all(err < tolerances(ws, tol)), err


def test_more_isobar_classes_than_a_table_holds():
    """700 mass bins of a freed isobar: several batches of one topology class."""
    edges = np.linspace(0.28, 2.2, 701)
    ws = []
    for lo, hi in zip(edges[:-1], edges[1:]):
        ow = O.wave(0, -1, 0, +1, 0, 0, 0, 0, O.MASSDEP_BINNED, 0.0, 0.0, (1, 2), 0, False, bounds=(lo, hi))
        kw = dict(J=0, P=-1, M=0, refl=+1, L=0, S=0, isobarJ=0, isobarL=0, massDependence="binned",
                  isobarMass=0.0, isobarWidth=0.0, isobarDaughters=(1, 2), bachelor=0, bounds=(lo, hi))
        ws.append((ow, kw))
    ws += waves()
    beam, fs, masses, mb = events(300, seed=5)
    ref = O.amplitudes([w for w, _ in ws], beam, fs, masses, mb, SPECIES)
    got = _amp(ws, masses, mb).amplitudes(beam, fs)
    # an event whose isobar mass lies within rounding of a bin edge may fall on either side
    bad = np.abs(got - ref) > TOL * 10 * np.maximum(1.0, np.abs(ref).max(axis=1, keepdims=True))
    assert bad.sum() <= 4
