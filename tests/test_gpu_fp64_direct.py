"""FP64 fits on singular likelihoods, and the direct form of the fit.

A saddle-point PSF is the same above and below focus, so at z = 0 its likelihood has a
stationary point without information on z.  A fit that starts or passes there turns
where the last bit of its sums sends it, so it is reproducible only while every sum keeps
its terms and their order.  FITS and ROWS are what the direct sums have always given for
the inputs below; the fits that converge elsewhere are the same to rounding in any order."""
import numpy as np
import pytest

import oracle as O
from common import OPTICS, astig_zernike, saddle_zernike, synth_rois, tetrapod_zernike
from test_gpu_detect import make_frames

pytestmark = pytest.mark.gpu

# z (um), its bound (um), status and evaluations
FITS = [
    (-0.19970104602695443, 0.016638993847324486, 1, 7), (0.16974123904608726, 0.02616474048673683, 1, 6),
    (-0.1685488860005075, 0.015351406061932414, 1, 5), (0.18806464993508948, 0.02710392162743825, 1, 11),
    (0.0007273366521684694, 6.004011414614182, 2, 50), (-0.15682476602211454, 0.031925979460055286, 1, 4),
    (-0.001339533556409942, 1.6443564896590719, 2, 50), (0.18253477653628855, 0.020162021662887837, 1, 5),
    (0.0007536336726759708, 5.272790717181967, 2, 50), (0.12975966379910064, 0.035771620405157675, 1, 16),
    (0.08357662514023503, 0.03154504312881521, 1, 5), (0.003549037035511772, 1.2410056484225542, 2, 50),
    (0.0008996491319224246, 4.985615929234063, 2, 50), (0.07174273801628166, 0.03419778400748874, 1, 6),
    (-0.16880599872712282, 0.028430746381224326, 1, 6), (0.0013196904596830448, 2.531581816730334, 2, 50),
    (0.15243049219854357, 0.021619609743372417, 1, 5), (-0.05737262764583669, 0.059574399116490845, 1, 5),
    (0.1034214490318836, 0.0288084320293854, 1, 12), (0.042923218267521976, 0.04663874554063745, 1, 6),
    (-0.08884516428674749, 0.041089313678738415, 1, 5), (0.13103448148134708, 0.034582769884401975, 1, 13),
    (0.051551375174228205, 0.09891047915559964, 1, 5), (-0.08199040710034976, 0.04053829897371737, 1, 5),
]
# frame, candidate, z (nm), its bound (nm) and fit status
ROWS = [
    (0, 59, -1049.3092355010988, 238.6978686415579, 2), (0, 299, -1119.317012085924, 300.1732190597447, 2),
    (1, 0, -143.60289299944407, 15.523646222656406, 1), (1, 13, 631.3688078974674, 9.184254623411901, 1),
    (1, 114, 908.1139008104396, 166.0551106553128, 1), (1, 321, -1171.2334514521199, 298.36261379065013, 1),
    (2, 0, 232.83453542329562, 11.712958615348722, 1), (2, 9, 838.1232996297389, 12.815021761018004, 1),
    (2, 72, -880.4499623315829, 156.8700826230962, 1), (3, 0, -210.10333834157132, 18.699853634827598, 1),
    (3, 7, 781.7445646451741, 11.937551952692907, 1), (3, 11, 643.9272784269681, 13.516346996455562, 1),
    (3, 100, -1170.985921537373, 190.5701941207722, 2), (3, 283, 1193.6075471348672, 309.38736857919184, 2),
    (4, 0, -0.004022509252221592, 386928.82678097434, 2), (4, 7, -532.1370155700525, 9.410984140586244, 1),
    (4, 11, -310.22232431114645, 13.812686037211437, 1), (4, 25, -412.89068802171175, 11.243036633199715, 1),
    (4, 248, -1160.2709091534869, 274.48348158092193, 2), (5, 0, -543.4788913645151, 10.947324944306482, 1),
    (5, 8, -114.32692908356226, 42.567855001469326, 1), (5, 13, -707.4590199848801, 15.157021123722558, 1),
]

# bounds of x, y, z, A and B at z = -0.4, -0.1, 0.2 and 0.7 um: saddle-point PSF at 16 px, tetrapod at 32
CURVES = [
    (0.007868305689257699, 0.007922431316582936, 0.01882294879580033, 0.04078725005365519, 2.4689880921895866),
    (0.005461397099965699, 0.005460581283804652, 0.03988488471251728, 0.0332764243269475, 1.9942218007470385),
    (0.005994802256941714, 0.006017662628759339, 0.022740739160277332, 0.034469653129589176, 2.0699863839537946),
    (0.013612420594048158, 0.013599980672872408, 0.028550771135346296, 0.07081896749957957, 4.3431914621636585),
    (0.014001708899311426, 0.00628155679810523, 0.049978319419405615, 0.04260048680692021, 2.2433393029672795),
    (0.00942903903344569, 0.006721259601168433, 0.034954083140892725, 0.03282525767306106, 1.7224912344024401),
    (0.006903436329235402, 0.009140991826916035, 0.025556560018025438, 0.0322894701249691, 1.693882068994273),
    (0.00776725138744841, 0.019450453318943642, 0.023130768564555176, 0.0427080773063525, 2.2490631311078926),
]


def test_fits_around_a_symmetric_focus(zpkg, ctx):
    """Starts at z = 0, 0.05 and -0.1 um: the depths and bounds of FITS to 1e-9, after as many evaluations."""
    zern = saddle_zernike()
    ref = O.OraclePSF(128, 0.11, 1.4, 0.66, 1.518, 1.518, 0.9, zern)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=128, **OPTICS), zern)
    rois, truth = synth_rois(ref.model, 16, 24, seed=5, zrange=0.2, photons=3000)
    init = truth.copy()
    init[:, :2] = 0
    init[:, 2] = np.array([0.0, 0.05, -0.1])[np.arange(24) % 3]
    prm = zpkg.PSF.fit_params(-1.0, 1.0, 0.88, max_iter=50, tol_xyz=1e-4, precision=zpkg.ZOLA_PREC_FP64)
    got, want = psf.fit(rois, init, prm), np.array(FITS)
    assert np.array_equal(got["status"], want[:, 2]) and np.array_equal(got["iters"], want[:, 3])
    assert np.allclose(got["theta"][:, 2], want[:, 0], rtol=1e-9, atol=0)
    assert np.allclose(got["crlb"][:, 2], want[:, 1], rtol=1e-9, atol=0)
    psf.close()


def test_movie_with_fits_that_do_not_converge(zpkg, ctx):
    """The rows of ROWS: the same candidates, statuses, depths and bounds (to 1e-9)."""
    zern = saddle_zernike()
    ref = O.OraclePSF(128, 0.11, 1.4, 0.66, 1.518, 1.518, 0.9, zern)
    fit = zpkg.PSF(ctx, zpkg.optics(size_fft=128, **OPTICS), zern)
    lib = zpkg.PSF(ctx, zpkg.optics(size_fft=128, kz_reset=True, **OPTICS), zern)
    frames = make_frames(ref.model, 112, 6, seed=18, emitters=5, R=48, zr=1.0)
    det = zpkg.Detector(lib, 112, 112, 24, -1.2, 1.2, 0.1, 0.1)
    got = zpkg.localize_frames(ctx, det, fit, frames, -1.2, 1.2, photon_threshold=300.0, max_iter=50,
                               precision=zpkg.ZOLA_PREC_FP64)
    want = np.array(ROWS)
    assert [(r["frame"], r["candidate"], r["fit_status"]) for r in got] == [(f, c, s) for f, c, _, _, s in ROWS]
    assert np.allclose(got["z_nm"], want[:, 2], rtol=1e-9, atol=0)
    assert np.allclose(got["crlb_z_nm"], want[:, 3], rtol=1e-9, atol=0)
    det.close()
    lib.close()
    fit.close()


def test_crlb_curves(zpkg, ctx):
    """CURVES to 1e-11: central differences of 0.5 nm magnify the models' rounding, 1e-16, by up to 1e7."""
    got = []
    for N, R, zern in ((64, 16, saddle_zernike()), (128, 32, tetrapod_zernike())):
        psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, **OPTICS), zern)
        got.append(psf.crlb_curve(R, [-0.4, -0.1, 0.2, 0.7]))
        psf.close()
    assert np.allclose(np.concatenate(got), CURVES, rtol=1e-11, atol=0)


@pytest.mark.parametrize("N,R,n", [(8, 4, 5), (16, 8, 3), (32, 14, 40), (64, 16, 1), (64, 30, 160), (128, 6, 37),
                                   (128, 18, 38), (128, 24, 149), (128, 48, 2), (256, 66, 3), (512, 20, 2)])
def test_direct_form_at_its_sizes(zpkg, ctx, N, R, n):
    """One evaluation converges nowhere, so every fit ends in the direct form (in clusters of eight, two or one
    CTA by the number of fits): likelihood and bounds at the start are those of the model.  Sums of up to 1e4
    terms of 64 bits, a Fisher matrix of condition 1e3: 1e-8.  The allocation-free form gives the same bits."""
    import torch
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, **OPTICS), astig_zernike() if N <= 64 else tetrapod_zernike())
    rng = np.random.default_rng(N + R)
    init = np.c_[rng.uniform(-0.1, 0.1, (n, 2)), rng.uniform(0.1, 0.4, n), rng.uniform(500, 3000, n), rng.uniform(5, 30, n)]
    psi, dpsi = psf.model(R, init[:, :3], derivs=True)
    A, B = init[:, 3, None, None], init[:, 4, None, None]
    mu = A * psi + B
    rois = rng.poisson(mu * rng.uniform(0.8, 1.25, mu.shape)).astype(np.float32)
    prm = zpkg.PSF.fit_params(-1.0, 1.0, 1.0, max_iter=1, tol_xyz=1e-9, precision=zpkg.ZOLA_PREC_FP64)
    got = psf.fit(rois, init, prm)
    d = rois.astype(np.float64)
    nll = (mu - d - d * np.log(np.where(d > 0, mu / np.where(d > 0, d, 1), 1))).sum((1, 2))
    J = np.concatenate([A[:, None] * dpsi, psi[:, None], np.ones_like(psi)[:, None]], 1).reshape(n, 5, -1)
    crlb = np.sqrt(np.linalg.inv((J / mu.reshape(n, 1, -1)) @ J.transpose(0, 2, 1)).diagonal(axis1=1, axis2=2))
    assert (got["status"] == 2).all() and (got["iters"] == 1).all() and np.array_equal(got["theta"], init)
    assert np.abs(got["nll"] - nll).max() <= 1e-8 * np.abs(mu).sum((1, 2)).max()
    if N > 8:  # (4 x 4 pixels hold next to nothing on z)
        assert np.allclose(got["crlb"], crlb, rtol=1e-8)
    t = lambda v, dt: torch.tensor(v, dtype=dt, device="cuda")  # noqa: E731
    out, c = (torch.zeros(n, 5, dtype=torch.float64, device="cuda") for _ in range(2))
    l = torch.zeros(n, dtype=torch.float64, device="cuda")
    zpkg.fit_noalloc_dev(psf, t(rois, torch.float32), t(init, torch.float64), prm, out, c, l, stream=ctx.stream)
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), got["theta"]) and np.array_equal(l.cpu().numpy(), got["nll"])
    assert np.array_equal(c.cpu().numpy(), got["crlb"], equal_nan=True)
    psf.close()
