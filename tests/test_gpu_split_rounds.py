"""GPU tests of how the round-based split fit spreads its ROIs over units and SMs, which
of them a round works through, and its eight-lane LM step."""
import numpy as np
import pytest

from common import astig_zernike, saddle_zernike, tetrapod_zernike
from test_gpu_flow import _job

pytestmark = pytest.mark.gpu

KEYS = ("theta", "crlb", "nll", "status", "iters")


def _same(a, b):
    return all(np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f") for k in KEYS)


@pytest.mark.parametrize("N,R,zern", [(64, 16, astig_zernike()), (128, 24, saddle_zernike()),
                                      (128, 40, tetrapod_zernike())])
def test_batch_sizes_pools_and_variance(zpkg, ctx, N, R, zern):
    """A ROI's fit does not depend on its unit, its neighbours or the pool: batches of one,
    about one ROI an SM and one unit an SM, and pools with fewer slots than ROIs equal the
    dataflow kernel's fit of the whole batch (which has the thread-a-slot LM step), bit for
    bit; with per-pixel variances as well."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    psf, rois, init, prm = _job(zpkg, ctx, N, R, zern, 4 * sms + 1, seed=300 + R + N)
    var = np.random.default_rng(R).uniform(0.5, 4.0, rois.shape).astype(np.float32)
    try:
        for scmos in (None, var):
            ctx.set_split_mode("flow")
            want = psf.fit(rois, init, prm, scmos=scmos)
            ctx.set_split_mode("staged")
            assert (want["status"] == 1).mean() > 0.8
            for n in (1, 2, sms - 1, sms, sms + 1, 2 * sms - 1, 2 * sms + 1, 4 * sms - 1, 4 * sms, 4 * sms + 1):
                got = psf.fit(rois[:n], init[:n], prm, scmos=None if scmos is None else scmos[:n])
                assert _same(got, {k: want[k][:n] for k in KEYS}), n
            for pool in (1, 4, sms + 4):
                ctx.set_pool(pool)
                assert _same(psf.fit(rois, init, prm, scmos=scmos), want), pool
                ctx.set_pool(0)
    finally:
        ctx.set_pool(0)
        ctx.set_split_mode("staged")
    psf.close()
