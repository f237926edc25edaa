"""GPU tests of the device memory that calls leave with a context."""
import numpy as np
import pytest

from common import OPTICS, astig_zernike
from test_oracle import drift_data

pytestmark = pytest.mark.gpu


def _kept(call, first):
    """Device bytes that `call` keeps, after `first` has loaded its kernels."""
    import torch
    first()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    call()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info(0)[0]


def test_drift_gives_its_buffers_back(zpkg):
    """A job of windows of 128 voxels needs 1.5 GB; the context keeps none of it (64 MB for what else may move)."""
    ctx = zpkg.Context(0)
    xyz, fr, cr, _, _ = drift_data(seed=3, nf=500, nbead=30, n_per=40, L=1500.0, Lz=300.0, vel=(0.02, -0.01, 0.005))
    job = lambda bins: zpkg.drift(ctx, xyz, fr, cr, pixel_nm=10.0, bins=bins, max_drift_um=1.28)  # noqa: E731
    assert _kept(lambda: job(6), lambda: job(2)) < 64 << 20
    ctx.close()
