"""The FFT screening of the detection against the direct correlation, bit for bit.

A detector with a threshold below 1e-3 takes the direct sum for every score, one
with a larger threshold screens by FFT and sums only the rows it returns.  Peaks
do not depend on the threshold except for the last test, so the rows of the first
whose score is above the second's threshold are the second's rows: the same
candidates in the same order with the same scores and offsets, exactly."""
import numpy as np
import pytest

from common import OPTICS, astig_zernike, tetrapod_zernike

pytestmark = pytest.mark.gpu


def frames_of(kind, n, SX, SY, seed):
    rng = np.random.default_rng(seed)
    f = rng.poisson(20.0, (n, SX, SY)).astype(np.float64)
    for k in range(n):
        for _ in range(3):
            a, b = rng.integers(0, SX - 6), rng.integers(0, SY - 6)
            f[k, a:a + 6, b:b + 6] += rng.poisson(60.0, (6, 6))
    if kind == "scaled":      # photons that are not whole numbers
        f = f * 0.47 - 1.3
    elif kind == "sparse":    # empty windows: the variance is zero, or one photon's
        f = rng.poisson(0.002, (n, SX, SY)).astype(np.float64)
    elif kind == "hot":       # a saturated pixel, and one far outside the range of a camera
        f[:, SX // 2, SY // 2] = 65535.0
        f[0, 3, 4] = 1e12
    elif kind == "nan":       # pixels that are not finite, in one of the frames
        f[0, SX // 3, SY // 2] = np.nan
        f[-1, SX // 3, SY // 2] = np.inf
    elif kind == "flat":      # a constant that is not exact in binary beside a pattern
        f[:, :, : SY // 2] = 0.1
    elif kind == "tiles":     # the same patch again and again: equal scores far apart
        t = f[:, : SX // 3, : SY // 3]
        f = np.tile(t, (1, 4, 4))[:, :SX, :SY].copy()
    elif kind == "mirror":    # equal scores next to each other
        f = f + f[:, ::-1, :]
    return f


CASES = [
    # lengths of the transforms: 50 px is the least, 64, 144 and 288 points, odd and unequal sides
    ("plain", 43, 43, 14, 64, -0.3, 0.3, 0.1), ("plain", 47, 61, 14, 64, -0.3, 0.3, 0.11),
    ("plain", 42, 60, 14, 64, -0.3, 0.3, 0.1), ("plain", 64, 64, 12, 64, -0.3, 0.3, 0.1),  # direct on both sides
    ("plain", 130, 130, 16, 64, -0.6, 0.6, 0.1), ("scaled", 131, 97, 24, 64, -0.4, 0.5, 0.1),
    ("plain", 268, 200, 40, 128, -0.5, 0.5, 0.1), ("scaled", 200, 269, 40, 128, -0.2, 0.2, 0.1),
    # one slice, two, three (the last pair has one)
    ("plain", 96, 96, 16, 64, 0.0, 0.1, 0.1), ("plain", 96, 96, 16, 64, 0.0, 0.2, 0.1),
    ("scaled", 96, 96, 16, 64, 0.0, 0.3, 0.1),
    # four passes, and the largest window
    ("plain", 540, 90, 30, 128, -0.1, 0.2, 0.1), ("plain", 200, 200, 96, 128, -0.1, 0.2, 0.1),
    # frames that the screening leaves to the direct sum, or that test its bound
    ("sparse", 100, 100, 20, 64, -0.3, 0.3, 0.1), ("hot", 100, 90, 20, 64, -0.3, 0.3, 0.1),
    ("nan", 100, 90, 20, 64, -0.3, 0.3, 0.1), ("flat", 100, 90, 20, 64, -0.3, 0.3, 0.1),
    ("tiles", 120, 120, 16, 64, -0.3, 0.3, 0.1), ("mirror", 100, 100, 16, 64, -0.3, 0.3, 0.1),
]


@pytest.mark.parametrize("kind,SX,SY,R,N,lo,hi,step", CASES)
def test_fft_screening_gives_the_direct_rows(zpkg, ctx, kind, SX, SY, R, N, lo, hi, step):
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, kz_reset=True, **OPTICS),
                   astig_zernike() if N == 64 else tetrapod_zernike())
    frames = frames_of(kind, 3, SX, SY, seed=SX + R)
    direct = zpkg.Detector(psf, SX, SY, R, lo, hi, step, 5e-4)
    fft = zpkg.Detector(psf, SX, SY, R, lo, hi, step, 0.1)
    want, n_want = direct.detect(frames, cap=20000)
    whole, n = fft.detect(frames, cap=20000)   # rows completed in list order
    best, _ = fft.detect(frames, cap=40)       # ranked by the screening, the best completed
    assert n_want.max() <= 20000
    for f in range(len(frames)):
        w = want[f][want[f][:, 0] > 0.1]
        assert n[f] == len(w)
        assert np.array_equal(whole[f], w, equal_nan=True)
        assert np.array_equal(best[f], w[:40], equal_nan=True)
    if kind not in ("nan", "sparse"):
        assert n.min() > 0
    direct.close()
    fft.close()
    psf.close()
