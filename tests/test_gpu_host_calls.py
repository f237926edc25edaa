"""GPU tests of host-buffer calls on device pointers, which the driver's copies take as well."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FITS = """
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


GRADIENT = """
import ctypes, sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
import __graft_entry__ as ge
from common import OPTICS
z = ge.load_package()
ctx = z.Context(0)
nz, nb, ns, R = 9, 2, 3, 16
psf = z.PSF(ctx, z.optics(size_fft=64, n_wat=1.4, **OPTICS), np.zeros(nz))
rng = np.random.default_rng(0)
zern = np.r_[0, 0, 0, rng.normal(0, 0.2, nz - 3)]
bead = np.zeros((nb, 3 + ns + 6))
bead[:, 3:3 + ns], bead[:, 3 + ns] = 9000, 80
cal = z.Calibration(psf, rng.poisson(200.0, (nb, ns, R, R)).astype(float), np.linspace(-0.3, 0.3, ns))
nll, gz, gs, gb = cal.backward(zern, 0.95, bead)
P = lambda a: ctypes.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)
data = cal._data(nz)
d_bead, d_gb = torch.tensor(bead, device="cuda"), torch.zeros(nb, 3 + ns + 6, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
f, g, s = np.zeros(1), np.zeros(nz), np.zeros(1)
L = z.lib()
assert L.zola_calib_backward(psf.h, ctypes.byref(data), P(zern), ctypes.c_double(0.95), P(d_bead), P(f), P(g), P(s), P(d_gb)) == 0
torch.cuda.synchronize()
assert f[0] == nll and np.array_equal(g, gz) and s[0] == gs and np.array_equal(d_gb.cpu().numpy(), gb)
assert L.zola_calib_forward(psf.h, ctypes.byref(data), P(zern), ctypes.c_double(0.95), P(d_bead), P(f), None) == 0
assert f[0] == cal.forward(zern, 0.95, bead)
print("FINE")
"""


def _run(script):
    r = subprocess.run([sys.executable, "-c", script.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "FINE" in r.stdout, r.stdout + r.stderr


def test_fits_on_device_pointers(zpkg):
    """Small and larger calls whose ROIs, starts or results are on the device: the results of host buffers."""
    _run(FITS)


def test_calibration_gradient_on_device_pointers(zpkg):
    """Bead parameters and their gradient on the device: those of host buffers."""
    _run(GRADIENT)
