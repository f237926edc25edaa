"""The FP64 model and fit through N-point FFTs in clusters of CTAs, at the sizes where
their tiles, windows and cluster shapes change, against direct sums in numpy.

Tolerance: the transforms and blurs are sums of at most D^2 W terms whose rounding grows
like the square root of their number times 2^-53, so relative to the largest value
1e-12 leaves a factor of ten."""
import numpy as np
import pytest

from common import OPTICS, astig_zernike, tetrapod_zernike

pytestmark = pytest.mark.gpu


def reference(N, R, zern, xyz, kz_reset, na, sigma=0.9, dx=0.11, lam=0.66, n=1.518):
    """psi (m, R, R) and dpsi (m, 3, R, R) by direct partial DFTs and a dense circular blur."""
    from math import factorial as f
    c = N / 2 - 0.5
    u = (np.arange(N) - c) / (N * dx)
    ring, rr = (na / lam) ** 2, u[:, None] ** 2 + u[None, :] ** 2
    disk = rr <= ring
    rho, th = np.sqrt(rr) * lam / na, np.arctan2(u[None, :] + 0 * u[:, None], u[:, None] + 0 * u[None, :])
    phase, k, order = np.zeros((N, N)), 0, 0
    while k < len(zern):
        for m in range(-order, order + 1, 2):
            if k < len(zern):
                am = abs(m)
                rad = sum((-1) ** q * f(order - q) / (f(q) * f((order + am) // 2 - q) * f((order - am) // 2 - q)) *
                          rho ** (order - 2 * q) for q in range((order - am) // 2 + 1))
                phase += zern[k] * np.where(rho < 1, rad * (np.cos(am * th) if m >= 0 else np.sin(am * th)), 0)
                k += 1
        order += 1
    q2 = (n / lam) ** 2 - rr
    kz = 2 * np.pi * np.sqrt(np.abs(q2)) * ((q2 > 0) | bool(kz_reset))
    W = 1 << (min(2 * R, N) - 1).bit_length()
    w = np.arange(W) - W // 2
    C = np.exp(2j * np.pi * (np.outer(w, np.arange(N) + N // 2) % N) / N)
    fr = np.where(np.arange(W) < W // 2, np.arange(W), np.arange(W) - W)
    g = np.exp(-0.5 * fr ** 2 / (W / (2 * np.pi * sigma)) ** 2)
    h = (g[None, :] * np.cos(2 * np.pi * np.outer(np.arange(W), np.arange(W)) / W)).sum(1) / W
    G = h[(np.arange(R)[:, None] - R // 2 - w[None, :]) % W]
    kx = 2 * np.pi * u
    psi, dpsi = [], []
    for x, y, z in xyz:
        p = kx[:, None] * x + kx[None, :] * y + phase
        Q = disk * (np.cos(p + kz * z) + 1j * np.sin(p + kz * z * (q2 > 0)))
        E = C @ Q @ C.T
        T = [np.abs(E) ** 2] + [2 * np.real(np.conj(E) * (C @ (1j * d * Q) @ C.T))
                                for d in (kx[:, None] + 0 * kz, kx[None, :] + 0 * kz, kz)]
        B = [G @ t @ G.T for t in T]
        sg, tot = np.where(B[0] < 0, -1, 1), np.abs(B[0]).sum()
        psi.append(np.abs(B[0]) / tot)
        dpsi.append([(sg * b - psi[-1] * (sg * b).sum()) / tot for b in B[1:]])
    return np.array(psi), np.array(dpsi)


@pytest.mark.parametrize("N,R,na,kz_reset", [
    (8, 4, 1.4, False), (16, 16, 1.4, False), (32, 8, 1.4, False), (32, 32, 1.4, False),  # one tile
    (64, 4, 1.4, False), (64, 16, 1.4, False), (64, 18, 1.4, True), (64, 64, 1.4, False),   # one CTA, two
    (128, 6, 1.4, False), (128, 16, 1.4, False), (128, 18, 1.2, False), (128, 50, 1.4, True),  # one, two, four
    (128, 30, 0.45, False), (128, 128, 1.4, False),                # fewer row tiles than CTAs; the whole grid
    (256, 10, 1.4, False), (256, 70, 1.3, False), (512, 34, 1.4, False), (1024, 12, 1.4, False)])
def test_fft_model_matches_direct_sums(zpkg, ctx, N, R, na, kz_reset):
    zern = astig_zernike() if N <= 64 else tetrapod_zernike()
    opt = dict(OPTICS, na=na)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, kz_reset=kz_reset, **opt), zern)
    rng = np.random.default_rng(N + R)
    xyz = rng.uniform(-1, 1, (3, 3)) * [0.2, 0.2, 0.8]
    want, dwant = reference(N, R, zern, xyz, kz_reset, na)
    psi, dpsi = psf.model(R, xyz, derivs=True)
    alone = psf.model(R, xyz[1:2])
    assert np.abs(psi - want).max() < 1e-12 * want.max()
    assert np.array_equal(alone[0], psi[1])  # neither the batch nor the derivatives change psi
    if not kz_reset:  # the derivatives assume the fit tables
        for q in range(3):
            assert np.abs(dpsi[:, q] - dwant[:, q]).max() < 1e-12 * np.abs(dwant[:, q]).max()
    psf.close()


@pytest.mark.parametrize("N,R,n", [(64, 16, 1), (64, 32, 7), (128, 16, 3), (128, 24, 300), (128, 48, 2), (256, 20, 2)])
def test_fp64_fit_does_not_depend_on_the_batch(zpkg, ctx, N, R, n):
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, **OPTICS), astig_zernike())
    rng = np.random.default_rng(R)
    truth = np.c_[rng.uniform(-0.1, 0.1, (n, 2)), rng.uniform(-0.4, 0.4, n), rng.lognormal(8, 0.3, n), np.full(n, 20.0)]
    rois = rng.poisson(truth[:, 3, None, None] * psf.model(R, truth[:, :3]) + 20.0).astype(np.float32)
    init = truth * [0, 0, 1, 1, 1] + [0, 0, 0.05, 0, 0]
    prm = zpkg.PSF.fit_params(-1, 1, R * 0.055, max_iter=40, tol_xyz=1e-4)
    a = psf.fit(rois, init, prm)
    order = rng.permutation(n)[: max(1, n // 2)]
    b = psf.fit(rois[order], init[order], prm)
    for k in a:
        assert np.array_equal(a[k][order], b[k])
    ok = a["status"] == 1
    assert ok.mean() > 0.8
    # the fits end at the optimum: within five standard errors of the truth
    assert (np.abs(a["theta"] - truth)[ok] < 5 * a["crlb"][ok] + 1e-9).mean() > 0.95
    psf.close()
