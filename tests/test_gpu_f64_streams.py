"""GPU tests of FP64 models and fits of small windows on several streams and under capture."""
import numpy as np
import pytest

from common import OPTICS, astig_zernike, saddle_zernike

pytestmark = pytest.mark.gpu

SIZES = [(64, 16), (64, 10), (32, 16), (128, 8)]


@pytest.mark.parametrize("N,R", SIZES)
def test_first_model_and_fit_of_a_context_under_capture(zpkg, ctx, N, R):
    """A context that has computed nothing yet records a model and a fit (its tables are ready; the kernels are
    loaded by another context): no allocation gets in the way, and the replays give the results of direct calls."""
    import torch
    n = 300
    rng = np.random.default_rng(N + R)
    init = np.c_[rng.uniform(-0.1, 0.1, (n, 2)), rng.uniform(0.1, 0.4, n), rng.uniform(800, 3000, n), rng.uniform(5, 30, n)]
    other = zpkg.PSF(ctx, zpkg.optics(size_fft=N, **OPTICS), astig_zernike())
    psi = other.model(R, init[:, :3])
    rois = rng.poisson(init[:, 3, None, None] * psi + init[:, 4, None, None]).astype(np.float32)
    prm = zpkg.PSF.fit_params(-1.0, 1.0, 1.0, max_iter=50, tol_xyz=1e-4, precision=zpkg.ZOLA_PREC_FP64)
    want = other.fit(rois, init, prm)
    fresh = zpkg.Context(0)
    psf = zpkg.PSF(fresh, zpkg.optics(size_fft=N, **OPTICS), astig_zernike())
    t = lambda v, dt=torch.float64: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    xyz, d_rois, d_init = t(np.ascontiguousarray(init[:, :3])), t(rois, torch.float32), t(init)
    out, theta = torch.zeros(n, R, R, dtype=torch.float64, device="cuda"), torch.zeros(n, 5, dtype=torch.float64, device="cuda")
    psf.model_dev(R, xyz[:0], out)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s = torch.cuda.current_stream().cuda_stream
        psf.model_dev(R, xyz, out, stream=s)
        psf.fit_dev(d_rois, d_init, prm, theta, stream=s)
    for _ in range(2):
        out.zero_()
        theta.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), psi) and np.array_equal(theta.cpu().numpy(), want["theta"])
    del g
    fresh.close()
    other.close()


@pytest.mark.parametrize("N,R", SIZES)
def test_models_and_fits_on_streams_at_once(zpkg, ctx, N, R):
    """Models and fits of one context on three streams, without a wait in between, beside models of a large window
    in the shared scratch: every result is that of a call by itself."""
    import torch
    n = 600
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, **OPTICS), saddle_zernike() if N == 128 else astig_zernike())
    large = zpkg.PSF(ctx, zpkg.optics(size_fft=128, **OPTICS), astig_zernike())
    rng = np.random.default_rng(7)
    t = lambda v, dt=torch.float64: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    prm = zpkg.PSF.fit_params(-1.0, 1.0, 1.0, max_iter=50, tol_xyz=1e-4, precision=zpkg.ZOLA_PREC_FP64)
    jobs = []
    for k in range(3):
        init = np.c_[rng.uniform(-0.1, 0.1, (n, 2)), rng.uniform(0.1, 0.4, n), rng.uniform(800, 3000, n),
                     rng.uniform(5, 30, n)]
        psi = psf.model(R, init[:, :3])
        rois = rng.poisson(init[:, 3, None, None] * psi + init[:, 4, None, None]).astype(np.float32)
        jobs.append((psi, psf.fit(rois, init, prm)["theta"], t(np.ascontiguousarray(init[:, :3])), t(rois, torch.float32),
                     t(init)))
    big = large.model(40, jobs[0][2].cpu().numpy()[:200])
    outs = [[(torch.zeros(n, R, R, dtype=torch.float64, device="cuda"), torch.zeros(n, 5, dtype=torch.float64, device="cuda"))
             for _ in jobs] for _ in range(3)]
    big_out, big_xyz = torch.zeros(200, 40, 40, dtype=torch.float64, device="cuda"), jobs[0][2][:200].contiguous()
    streams = [torch.cuda.Stream() for _ in jobs]
    torch.cuda.synchronize()
    for rep in range(3):
        for (_, _, xyz, rois, init), (psi, theta), s in zip(jobs, outs[rep], streams):
            psf.model_dev(R, xyz, psi, stream=s.cuda_stream)
            psf.fit_dev(rois, init, prm, theta, stream=s.cuda_stream)
        large.model_dev(40, big_xyz, big_out, stream=ctx.stream)
    torch.cuda.synchronize()
    for rep in outs:
        for (psi, theta, *_), (p, th) in zip(jobs, rep):
            assert np.array_equal(p.cpu().numpy(), psi) and np.array_equal(th.cpu().numpy(), theta)
    assert np.array_equal(big_out.cpu().numpy(), big)
    psf.close()
    large.close()
