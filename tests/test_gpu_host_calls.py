"""GPU test of a host-buffer fit on device pointers, which the driver's copies take as well."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
import __graft_entry__ as ge
from common import OPTICS, astig_zernike
z = ge.load_package()
ctx = z.Context(0)
psf = z.PSF(ctx, z.optics(size_fft=64, **OPTICS), astig_zernike())
R, rng = 16, np.random.default_rng(0)
prm = z.PSF.fit_params(-1, 1, 1, max_iter=30, tol_xyz=1e-4, precision=z.ZOLA_PREC_SPLIT)
P = lambda t: ctypes.c_void_p(t.data_ptr())
for n in (5, 1500):
    init = np.c_[np.zeros((n, 2)), np.full(n, 0.2), np.full(n, 1000.0), np.full(n, 20.0)]
    rois = rng.poisson(1000 * psf.model(R, [[0, 0, 0.25]])[0] + 20, (n, R, R)).astype(np.float32)
    want = psf.fit(rois, init, prm)
    hr, hi, ho = torch.tensor(rois), torch.tensor(init), torch.zeros(n, 5, dtype=torch.float64)
    for where in range(1, 8):  # which of the three are on the device
        a, b, c = ((t.cuda() if where >> k & 1 else t.clone()) for k, t in enumerate((hr, hi, ho)))
        torch.cuda.synchronize()
        rc = z.lib().zola_fit_batch(ctx.h, psf.h, R, P(a), P(b), n, ctypes.byref(prm), P(c), None, None, None, None)
        torch.cuda.synchronize()
        assert rc == 0 and np.array_equal(c.cpu().numpy(), want["theta"]), (n, where)
print("FINE")
"""


def test_fits_on_device_pointers(zpkg):
    """Small and larger calls whose ROIs, starts or results are on the device: the results of host buffers."""
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "FINE" in r.stdout, r.stdout + r.stderr
