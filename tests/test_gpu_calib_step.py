"""One Levenberg-Marquardt step of the calibration against numpy: the Gauss-Newton matrix
from central differences of the forward model, the gradient from the adjoint, and the
damped solve; at the sizes where the kernels' blocks change (Gram tiles of four
directions, 128 of them a pass; 32-column blocks of the factorisation, 256 rows staged;
window and cluster shapes).

Tolerance: central differences with a relative step h have errors h^2 / 6 + 1e-16 / h,
at most 1e-9 of a tangent for h = 1e-5; the damping bounds the matrix's condition, so the
step is compared within 1e-4 of its largest entry per parameter group."""
import numpy as np
import pytest

from common import OPTICS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R,nz,nb,ns,fit_sigma", [
    (32, 8, 4, 1, 1, True), (64, 8, 7, 1, 2, False), (64, 16, 12, 2, 3, True), (128, 18, 15, 2, 5, True),
    (64, 32, 9, 1, 3, True),
    (64, 10, 45, 2, 12, True),   # 89 parameters
    (64, 8, 16, 3, 85, True),    # 296 parameters: two staged row blocks
    (64, 8, 100, 1, 4, False),   # 108 directions: three passes of Gram tiles (and too few pixels for a good step)
    (64, 20, 90, 1, 16, True),   # 98 directions, a step that is taken
])
def test_one_step_matches_numpy(zpkg, ctx, N, R, nz, nb, ns, fit_sigma):
    rng = np.random.default_rng(nz + ns)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, n_wat=1.4, **OPTICS), np.zeros(nz))
    dz = np.linspace(-0.5, 0.5, ns) if ns > 1 else np.array([0.2])
    zt = rng.normal(0, 0.2, nz)
    zt[:3] = 0
    pb = 3 + ns + 6
    bead = np.zeros((nb, pb))
    bead[:, :3] = rng.uniform(-0.03, 0.03, (nb, 3))
    bead[:, 3:3 + ns] = rng.uniform(9000, 12000, (nb, ns))
    bead[:, 3 + ns] = 80.0
    shape = (nb, ns, R, R)
    _, mu = zpkg.Calibration(psf, np.ones(shape), dz).forward(zt, 1.0, bead, model=True)
    cal = zpkg.Calibration(psf, rng.poisson(mu).astype(float), dz)
    z0, s0, b0 = zt * 0.97, 0.98, bead.copy()
    b0[:, 3:3 + ns] *= 1.02

    def theta(z, s, b):
        return np.concatenate([z[3:], [s] if fit_sigma else [], b.ravel()])

    def split(t):
        k = nz - 3 + int(fit_sigma)
        return np.concatenate([z0[:3], t[:nz - 3]]), (t[nz - 3] if fit_sigma else s0), t[k:].reshape(nb, pb)

    nll0, gz, gs, gb = cal.backward(z0, s0, b0)
    g = np.concatenate([gz[3:], [gs] if fit_sigma else [], gb.ravel()])
    t0 = theta(z0, s0, b0)
    mu0 = cal.forward(z0, s0, b0, model=True)[1].ravel()
    J = np.empty((mu0.size, len(t0)))
    for p in range(len(t0)):
        h = 1e-5 * max(1.0, abs(t0[p]))
        up, dn = t0.copy(), t0.copy()
        up[p] += h
        dn[p] -= h
        J[:, p] = (cal.forward(*split(up), model=True)[1].ravel() - cal.forward(*split(dn), model=True)[1].ravel()) / (2 * h)
    H = (J / mu0[:, None]).T @ J
    lam = 1e-3
    step = -np.linalg.solve(H + np.diag(lam * np.maximum(np.diag(H), 1e-12)), g)
    z1, s1, b1, nll1, it = cal.fit(z0, s0, b0, max_iter=1, fit_sigma=fit_sigma)
    assert it == 1
    got = theta(z1, s1, b1) - t0
    if cal.forward(*split(t0 + step)) > nll0:  # a step that raises the likelihood is not taken
        assert nll1 == nll0 and not got.any()
        return
    assert nll1 < nll0
    k = nz - 3 + int(fit_sigma)
    bg, bw = got[k:].reshape(nb, pb), step[k:].reshape(nb, pb)
    groups = [(got[:nz - 3], step[:nz - 3]), (got[nz - 3:k], step[nz - 3:k])]
    groups += [(bg[:, a:b], bw[:, a:b]) for a, b in ((0, 3), (3, 3 + ns), (3 + ns, pb))]
    for a, b in groups:
        if b.size:
            assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()
    psf.close()
