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


@pytest.mark.parametrize("derivs", [False, True])
def test_large_model_calls_give_their_buffers_back(zpkg, derivs):
    """Models of 0.6 GB: the same as in small calls, and no more is kept than a call of 256 MB keeps (in steps of
    64 MB, and as much for what else may move)."""
    ctx = zpkg.Context(0)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=64, **OPTICS), astig_zernike())
    xyz = np.random.default_rng(1).uniform(-0.3, 0.3, (73000 // (4 if derivs else 1), 3))
    got = []
    kept = _kept(lambda: got.append(psf.model(32, xyz, derivs=derivs)), lambda: psf.model(32, xyz[:10], derivs=derivs))
    assert kept < 384 << 20
    pick = np.r_[0:7, len(xyz) - 7:len(xyz)]
    few, many = psf.model(32, xyz[pick], derivs=derivs), got[0]
    for a, b in zip(few, many) if derivs else [(few, many)]:
        assert np.array_equal(a, b[pick])
    ctx.close()


def test_detection_without_room_for_the_spectra(zpkg):
    """A frame of 1200 x 1200 against 40 slices: 1.1 GB with the FFT correlation, 0.6 without.  With 0.9 GB left the
    rows are those of a detection with all the memory it wants."""
    import torch
    ctx = zpkg.Context(0)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=128, kz_reset=True, **OPTICS), astig_zernike())
    frames = np.random.default_rng(2).poisson(20.0, (1, 1200, 1200)).astype(float)
    frames[:, 300:306, 500:506] += 300
    det = zpkg.Detector(psf, 1200, 1200, 40, -2.0, 2.0, 0.1, 0.1)
    want, n = det.detect(frames, cap=500)
    ctx2 = zpkg.Context(0)
    psf2 = zpkg.PSF(ctx2, zpkg.optics(size_fft=128, kz_reset=True, **OPTICS), astig_zernike())
    det2 = zpkg.Detector(psf2, 1200, 1200, 40, -2.0, 2.0, 0.1, 0.1)
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info(0)[0] - (900 << 20), dtype=torch.uint8, device="cuda")
    try:
        got, m = det2.detect(frames, cap=500)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert n[0] == m[0] > 0 and np.array_equal(want[0], got[0])
    det.close()
    det2.close()
    ctx.close()
    ctx2.close()
