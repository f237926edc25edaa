"""GPU test of large calls on pageable host memory, whose copies run on several threads."""
import numpy as np
import pytest

from common import astig_zernike
from test_gpu_flow import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4095, 4096, 4097, 12801])
def test_pageable_and_pinned_calls_agree(zpkg, ctx, n):
    """Around 4 MB of ROIs (4,096 of 16 x 16) and with a ragged last segment: the same fits
    and models, bit for bit, as from pinned memory and in small calls; twice, so that the
    buffers are used again."""
    import torch
    psf, few, few_init, prm = _job(zpkg, ctx, 64, 16, astig_zernike(), 500, seed=77)
    pick = np.random.default_rng(n).integers(0, 500, n)
    rois, init = few[pick], few_init[pick]
    pinned = torch.from_numpy(rois).pin_memory().numpy()
    for _ in range(2):
        a, b = psf.fit(rois, init, prm), psf.fit(pinned, init, prm)
        for k in ("theta", "crlb", "nll", "status", "iters"):
            assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k
    xyz = init[:, :3]
    psi, dpsi = psf.model(16, xyz, derivs=True)
    parts = [psf.model(16, xyz[k:k + 500], derivs=True) for k in range(0, n, 500)]
    assert np.array_equal(psi, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(dpsi, np.concatenate([p[1] for p in parts]))
    psf.close()
