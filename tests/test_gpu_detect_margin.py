"""Detection beside a dark margin.

The columns within half a ROI of the border hold no candidates, but the three next to the
inner part are compared with those there.  Where the window of such a pixel is dark but for
a trace, 1e-18 of the brightest pixel of the frame here, its score from the FFT correlation
is that pixel's rounding."""
import numpy as np
import pytest

from common import OPTICS, astig_zernike

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,R,noise", [(64, 16, 1.0), (90, 20, 3.0)])
def test_candidates_beside_a_dark_margin(zpkg, ctx, S, R, noise):
    """One candidate a frame at the first inner column: the rows of a screened detection are those of direct
    sums (a threshold below 1e-3), bit for bit."""
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=64, kz_reset=True, **OPTICS), astig_zernike())
    rng = np.random.default_rng(S)
    n = 48
    frames = noise * rng.uniform(0, 1, (n, S, S))
    frames[:, :, :R] = 0
    frames[:, :, :R - 2] = 1e-12 * (rng.uniform(size=(n, S, R - 2)) < 0.05)
    frames[:, S // 2 - 7:S // 2 + 8, R - 2:R] = -1
    frames[:, :, 2 * R + 8:] = 1e6 * rng.uniform(0.5, 1, (n, S, S - 2 * R - 8))
    direct = zpkg.Detector(psf, S, S, R, 0.0, 0.1, 0.1, 5e-4)
    screened = zpkg.Detector(psf, S, S, R, 0.0, 0.1, 0.1, 2e-3)
    want, _ = direct.detect(frames, cap=20000)
    got, counts = screened.detect(frames, cap=20000)
    beside = 0
    for f in range(n):
        w = want[f][want[f][:, 0] > 2e-3]
        beside += (w[:, 3] == R // 2).sum()
        assert counts[f] == len(w) and np.array_equal(got[f], w)
    assert beside > n // 4
    direct.close()
    screened.close()
    psf.close()
