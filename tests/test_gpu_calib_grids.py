"""The calibration's gradient on the smallest pupil grids, against central differences of its
likelihood.

Tolerance: a relative step h has errors of h^2 of the likelihood's third derivative and of
1e-16 nll / h; with h = 1e-4 of a parameter's scale both stay below 1e-5 of the largest
gradient of its kind."""
import numpy as np
import pytest

from common import OPTICS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R", [(4, 4), (8, 4), (8, 8), (16, 6), (16, 16)])
def test_gradient_matches_differences(zpkg, ctx, N, R):
    nz, nb, ns = 7, 2, 3
    rng = np.random.default_rng(10 * N + R)
    psf = zpkg.PSF(ctx, zpkg.optics(size_fft=N, n_wat=1.4, **OPTICS), np.zeros(nz))
    dz = np.linspace(-0.4, 0.5, ns)
    zern = np.r_[0, 0, 0, rng.normal(0, 0.3, nz - 3)]
    bead = np.zeros((nb, 3 + ns + 6))
    bead[:, :3] = rng.uniform(-0.05, 0.05, (nb, 3))
    bead[:, 3:3 + ns] = rng.uniform(9000, 12000, (nb, ns))
    bead[:, 3 + ns] = 80.0
    _, mu = zpkg.Calibration(psf, np.ones((nb, ns, R, R)), dz).forward(zern, 1.0, bead, model=True)
    cal = zpkg.Calibration(psf, rng.poisson(1.1 * mu).astype(float), dz)
    _, gz, gs, gb = cal.backward(zern, 0.95, bead)

    def slope(step, h):
        up, dn = (cal.forward(zern + s * step.get("z", 0), 0.95 + s * step.get("s", 0), bead + s * step.get("b", 0))
                  for s in (1, -1))
        return ((up[0] if isinstance(up, tuple) else up) - (dn[0] if isinstance(dn, tuple) else dn)) / (2 * h)

    h, e = 1e-4, np.eye(nz)
    want = np.array([slope({"z": h * e[i]}, h) for i in range(3, nz)])
    assert np.abs(gz[3:] - want).max() <= 1e-5 * np.abs(want).max() and (gz[:3] == 0).all()
    assert abs(gs - slope({"s": h}, h)) <= 1e-5 * max(abs(gs), 1.0)
    for cols in ((0, 1, 2), range(3, 3 + ns), (3 + ns,)):
        step = h if cols[0] == 0 else 1.0 if cols[0] == 3 else 1e-2
        got, want = np.zeros((nb, len(cols))), np.zeros((nb, len(cols)))
        for b in range(nb):
            for k, c in enumerate(cols):
                d = np.zeros_like(bead)
                d[b, c] = step
                got[b, k], want[b, k] = gb[b, c], slope({"b": d}, step)
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), cols
    psf.close()
