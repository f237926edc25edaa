"""The allocation-free fit on pupil grids that the process has not fitted before.  Collected last on purpose."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
import __graft_entry__ as ge
from common import OPTICS, astig_zernike
z = ge.load_package()
ctx = z.Context(0)
prm = z.PSF.fit_params(-1.0, 1.0, 1.0, max_iter=20, tol_xyz=1e-4, precision=z.ZOLA_PREC_FP64)
n = 2000

def job(N, R):
    psf = z.PSF(ctx, z.optics(size_fft=N, **OPTICS), astig_zernike())
    psf.model_dev(R, torch.zeros(0, 3, dtype=torch.float64, device="cuda"), torch.zeros(1, device="cuda"))  # tables
    rng = np.random.default_rng(N)
    rois = torch.tensor(rng.poisson(20.0, (n, R, R)), dtype=torch.float32, device="cuda")
    init = torch.tensor(np.c_[np.zeros((n, 2)), np.full(n, 0.2), np.full(n, 500.0), np.full(n, 20.0)], device="cuda")
    out = torch.zeros(n, 5, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return lambda s=None: z.fit_noalloc_dev(psf, rois, init, prm, out, stream=s or ctx.stream), out

first, _ = job(64, 16)
first()
torch.cuda.synchronize()
kept = []
for N, R in ((8, 4), (16, 6), (32, 8), (128, 12), (256, 10), (512, 6)):
    call, out = job(N, R)
    free = torch.cuda.mem_get_info(0)[0]
    call()
    torch.cuda.synchronize()
    kept.append((N, free - torch.cuda.mem_get_info(0)[0]))
print("KEPT", kept)
"""


def test_every_grid_is_ready_after_the_first_call(zpkg):
    """A process's first call is on one pupil grid; then the first call on each other one takes no device memory."""
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    kept = eval(r.stdout.split("KEPT")[1])
    print(kept)
    assert all(b == 0 for _, b in kept), kept
