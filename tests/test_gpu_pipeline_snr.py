"""The pipeline's test of which candidates are fitted, at the last bit of getAandB's background."""
import numpy as np
import pytest

import oracle as O
from common import OPTICS, astig_zernike
from test_gpu_detect import make_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scmos", [False, True])
def test_candidates_on_the_edge_of_max_snr(zpkg, ctx, scmos):
    """The best candidate of a frame is fitted with max_snr one bit below its maxPatch / B and not with max_snr equal to
    it, B added up pixel after pixel as getAandB does (LocalizationPipeline.java:1119-1162)."""
    S, R = 96, 16
    zern = astig_zernike()
    lib = zpkg.PSF(ctx, zpkg.optics(size_fft=64, kz_reset=True, **OPTICS), zern)
    fit = zpkg.PSF(ctx, zpkg.optics(size_fft=64, **OPTICS), zern)
    ref = O.OraclePSF(64, 0.11, 1.4, 0.66, 1.518, 1.518, 0.9, zern)
    frames = make_frames(ref.model, S, 12, seed=31, emitters=4, R=32) * 0.4713 + 0.1
    det = zpkg.Detector(lib, S, S, R, -0.6, 0.6, 0.1, 0.1)
    img = det.library()[1]
    kw = dict(photon_threshold=100.0, precision=1, max_iter=40)
    if scmos:
        rng = np.random.default_rng(4)
        adu = frames.astype(np.float32)
        off, gain, var = np.zeros((S, S)), np.ones((S, S)), rng.uniform(0.5, 3.0, (S, S))
        det_img = np.maximum(adu.astype(float) + var[0, 0], 0)
        fit_img, sub = adu.astype(float) + var, var
        run = lambda f, snr: zpkg.localize_frames_scmos(ctx, det, fit, adu[f:f + 1], off, gain, var, -0.6, 0.6,  # noqa: E731
                                                        max_snr=snr, **kw)
    else:
        det_img = fit_img = frames
        sub = np.zeros((S, S))
        run = lambda f, snr: zpkg.localize_frames(ctx, det, fit, frames[f:f + 1], -0.6, 0.6, max_snr=snr, **kw)  # noqa: E731
    rows, _ = det.detect(det_img, cap=1)
    tested = 0
    for f in range(len(frames)):
        r, i, j = (int(v) for v in rows[f][0, 1:4])
        if not (R // 2 + 1 < min(i, j) and max(i, j) < S - R // 2 - 1):
            continue
        at = np.s_[i - R // 2:i + R // 2, j - R // 2:j + R // 2]
        patch = (fit_img[f][at] - sub[at]).ravel()
        low = img[r].ravel() < img[r].max() * 0.1
        B = 0.0
        for x in patch[low]:
            B += x
        snr = patch.max() / (B / low.sum())
        fitted = [0 in run(f, s)["candidate"] for s in (np.nextafter(snr, 0), snr)]
        if 0 in run(f, 1.0)["candidate"]:  # (a fit that the pipeline accepts)
            assert fitted == [True, False], f
            tested += 1
    assert tested >= 6
    det.close()
    lib.close()
    fit.close()
