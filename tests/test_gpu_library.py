"""GPU test of a detector's library images (direct sums in a fixed order)."""
import numpy as np
import pytest

import oracle as O
from common import OPTICS, astig_zernike, saddle_zernike, tetrapod_zernike

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R,zern,kz_reset", [(32, 4, astig_zernike(), True), (64, 15 * 2, astig_zernike(), True),
                                               (64, 64, saddle_zernike(), False), (128, 18, saddle_zernike(), True),
                                               (128, 40, tetrapod_zernike(), True)])
def test_library_images_match_the_model(zpkg, ctx, N, R, zern, kz_reset):
    """The images are the oracle's FP64 model at each depth: sums of D, D, W and W terms in
    64 bits (phases of some 100 rad) stay within 1e-12 of an image's maximum.  A second
    detector gives the same bits, and the FFT form of the model agrees as closely."""
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, kz_reset=kz_reset, **OPTICS), zern)
    ref = O.OraclePSF(N, 0.11, 1.4, 0.66, 1.518, 1.518, 0.9, zern, gauss_f32=False, kz_reset=kz_reset)
    a, b = (zpkg.Detector(psf, 96, 96, R, -0.65, 0.6, 0.1) for _ in range(2))
    z, img = a.library()
    assert len(z) == 13
    xyz = np.c_[np.zeros((len(z), 2)), z]
    for want in (np.stack([ref.model(R, p)[0] for p in xyz]), psf.model(R, xyz)):
        assert np.abs(img - want).max() <= 1e-12 * want.max()
    assert np.array_equal(img, b.library()[1])
    a.close(); b.close(); psf.close()
