"""How a split fit waits, in processes that ask the driver for waits of a kind."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, sys, time
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0 and cuda.cuDevicePrimaryCtxSetFlags_v2(0, {flags}) == 0
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
import __graft_entry__ as ge
from common import OPTICS, tetrapod_zernike
z = ge.load_package()
ctx = z.Context(0)
psf = z.PSF(ctx, z.optics(size_fft=128, **OPTICS), tetrapod_zernike())
n, R = 8000, 40
rng = np.random.default_rng(1)
init = np.c_[np.zeros((n, 2)), np.full(n, 0.2), np.full(n, 3000.0), np.full(n, 30.0)]
psi = psf.model(R, [[0.02, -0.01, 0.25]])[0]
rois = torch.tensor(rng.poisson(3000 * psi + 30, (n, R, R)), dtype=torch.float32, device="cuda")
init = torch.tensor(init, device="cuda")
out = torch.zeros(n, 5, dtype=torch.float64, device="cuda")
prm = z.PSF.fit_params(-1.0, 1.0, 2.2, max_iter=50, tol_xyz=1e-9, precision=z.ZOLA_PREC_SPLIT)
fit = lambda: psf.fit_dev(rois, init, prm, out)
fit()
wall, cpu = time.perf_counter(), time.process_time()
for _ in range(4):
    fit()
wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
print("SHARE", cpu / wall, wall)
"""


def _share(flags):
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT, flags=flags)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
    return float(r.stdout.split("SHARE")[1].split()[0])


def test_blocking_waits_leave_the_core(zpkg):
    """With cudaDeviceScheduleBlockingSync (4) the calling thread sleeps through most of a fit of some 100 ms: less
    than half of the time on a core, where launching its kernels takes a tenth."""
    assert _share(4) < 0.5
