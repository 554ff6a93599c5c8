"""Staging of the ptychography windows: even and odd columns, even- and odd-width objects,
windows inside, over an edge and outside the object, one sweep against the oracle with the
per-iterate bound of tests/test_gpu_ptycho.py."""
import numpy as np
import pytest

from oracle import ptycho_oracle as PO
from tests.test_gpu_ptycho import STEP_BOUND, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rows,cols", [(64, 150, 150), (64, 150, 151), (128, 300, 301), (128, 256, 258)])
@pytest.mark.parametrize("first", [0, 400])
def test_windows_match_oracle(cdx, n, rows, cols, first):
    from cdixx_gb300 import ptycho
    prm = PO.PtyParams(lam=0.5, d=2e5, dpupil=2e3, pixelsize=20.0, pupil_size=n * 0.6, exposure=1.0, mpie=True)
    rng = np.random.default_rng(n + cols)
    truth = (0.5 + rng.random((rows, cols))).astype(np.complex64)
    probe = PO.angular_spectrum(PO.pupil_func(n, n, prm.pupil_size), prm.lam, prm.dpupil, prm.resolution(n))
    # columns: even, odd, flush with either edge, over the left and the right edge
    sy = np.array([20, 21, 0, cols - n, -n // 3, cols - n // 2, 33], np.float32)
    sx = np.array([10, 31, rows - n, 0, 12, 40, -n // 4], np.float32)
    pats = PO.simulate_patterns(truth, probe, sx, sy)
    pats = (pats / pats.max() * 0.9).astype(np.float32)
    obj0 = np.exp(2j * np.pi * rng.random((rows, cols))).astype(np.complex64)
    c = {"obj0": obj0, "probe0": probe, "pats": pats, "scanx": sx, "scany": sy}
    orders = np.array([rng.permutation(len(sx))], np.int32)
    with make(ptycho, c, prm) as t:
        t.iterate(1, first_iter=first, orders=orders)
        O, _pupil, P = PO.iterate(obj0, probe, pats, sx, sy, 1, prm, orders, start_iter=first)
        assert PO.rel_err(t.objectWave, O) < STEP_BOUND
        assert PO.rel_err(t.probe, P) < STEP_BOUND
