"""GPU test of the calibration on beads whose blur matrices stay in global memory."""
import numpy as np
import pytest

from common import OPTICS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R,nz,nb,ns", [(128, 34, 12, 1, 2), (128, 40, 15, 1, 3), (128, 40, 15, 2, 3), (64, 60, 12, 1, 2),
                                          (128, 96, 12, 1, 1)])
def test_gradient_matches_central_differences(zpkg, ctx, N, R, nz, nb, ns):
    """The adjoint's derivative along a direction in every parameter group against the forward
    model's central difference, whether the parameters before the matrices are odd or even
    in number.  The step h = 1e-5 of each parameter's scale leaves errors h^2 / 6 and
    1e-16 |nll| / h of the derivative: 1e-4 of it (or of one photon) covers both."""
    rng = np.random.default_rng(R + nz + ns)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, n_wat=1.4, **OPTICS), np.zeros(nz))
    dz = np.linspace(-0.3, 0.3, ns) if ns > 1 else np.array([0.2])
    z = rng.normal(0, 0.2, nz)
    z[:3] = 0
    pb = 3 + ns + 6
    bead = np.zeros((nb, pb))
    bead[:, :3] = rng.uniform(-0.03, 0.03, (nb, 3))
    bead[:, 3:3 + ns] = rng.uniform(9000, 12000, (nb, ns))
    bead[:, 3 + ns] = 40.0
    _, mu = zpkg.Calibration(psf, np.ones((nb, ns, R, R)), dz).forward(z, 1.0, bead, model=True)
    cal = zpkg.Calibration(psf, rng.poisson(mu).astype(float), dz)
    z0, s0, b0 = z * 0.9, 0.95, bead.copy()
    b0[:, 3:3 + ns] *= 1.05
    _, gz, gs, gb = cal.backward(z0, s0, b0)
    nll = lambda z, s, b: cal.forward(z, s, b)  # noqa: E731
    h = 1e-5
    groups = [("z", rng.normal(0, 1, nz) * (np.arange(nz) > 2), 0.0, 0 * bead), ("sigma", 0 * z, 1.0, 0 * bead)]
    for name, a, b, scale in (("xyz", 0, 3, 0.1), ("photons", 3, 3 + ns, 1e4), ("background", 3 + ns, 4 + ns, 40.0)):
        d = np.zeros((nb, pb))
        d[:, a:b] = rng.normal(0, scale, (nb, b - a))
        groups.append((name, 0 * z, 0.0, d))
    for name, dzv, ds, db in groups:
        want = (nll(z0 + h * dzv, s0 + h * ds, b0 + h * db) - nll(z0 - h * dzv, s0 - h * ds, b0 - h * db)) / (2 * h)
        got = gz @ dzv + gs * ds + (gb * db).sum()
        assert abs(got - want) <= 1e-4 * max(abs(want), 1.0) + 1e-15 * abs(nll(z0, s0, b0)) / h, name
    psf.close()
