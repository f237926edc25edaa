"""GPU test of split fits on a caller's streams: the stream is idle when a call returns, so
that the context's next call may be on another one."""
import numpy as np
import pytest

from common import astig_zernike, saddle_zernike, tetrapod_zernike
from test_gpu_flow import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 700])
def test_alternating_streams(zpkg, ctx, n):
    """Fits of three classes, alternating between two non-blocking streams without a wait in between, and
    now and then followed by another user of the context's scratch (FP64 models on the other stream): the same
    results, bit for bit, as host calls one after the other.  A stream has nothing left to do after its fit."""
    import torch
    jobs = [_job(zpkg, ctx, N, R, z, n, seed=40 + R) for N, R, z in
            ((64, 16, astig_zernike()), (128, 24, saddle_zernike()), (128, 40, tetrapod_zernike()))]
    want = [psf.fit(rois, init, prm) for psf, rois, init, prm in jobs]
    t = lambda v, dt: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    dev = [(t(rois, torch.float32), t(init, torch.float64)) for _, rois, init, _ in jobs]
    outs = [[[torch.zeros(n, 5, dtype=torch.float64, device="cuda"), torch.zeros(n, 5, dtype=torch.float64, device="cuda"),
              torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"),
              torch.zeros(n, dtype=torch.int32, device="cuda")] for _ in jobs] for _ in range(4)]
    xyz = [init[:, :3].contiguous() for _, init in dev]
    psi = [torch.zeros(n, R, R, dtype=torch.float64, device="cuda") for R in (16, 24, 40)]
    s = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for rep in range(4):
        for c, (psf, rois, _, prm) in enumerate(jobs):
            a, b = s[(rep + c) % 2], s[(rep + c + 1) % 2]
            psf.fit_dev(*dev[c], prm, *outs[rep][c], stream=a.cuda_stream)
            assert a.query()
            if c == rep % 3:
                psf.model_dev(rois.shape[1], xyz[c], psi[c], stream=b.cuda_stream)
                b.synchronize()
    torch.cuda.synchronize()
    for got in outs:
        for w, o in zip(want, got):
            for k, v in zip(("theta", "crlb", "nll", "status", "iters"), o):
                assert np.array_equal(v.cpu().numpy(), w[k], equal_nan=w[k].dtype.kind == "f"), k
    for psf, *_ in jobs:
        psf.close()
