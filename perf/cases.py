"""What is timed: the calls a localization program makes, at the sizes it makes them.

A case is a dict of plain values.  ``listed()`` names the representative ones and
``draw(rng)`` gives more of the same ranges; ``prepare`` makes the inputs on the
seed, ``run`` makes one call through the package's public entry points,
``work`` counts the bytes and operations that the call cannot do without, and
``exact`` computes the same outputs in 64 bits with plain torch and numpy.

The context, the PSFs and the detectors are made once per optical set-up and
kept for the whole process, as a program keeps its calibration while frames and
ROIs stream past; every input comes from the seed.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TWO_PI = 2 * math.pi
DX = 0.11
OPT = dict(xystep=DX, na=1.4, wavelength=0.66, n_oil=1.518)
F64, C128 = torch.float64, torch.complex128


def _pkg():
    """The package directory zola-3d_b200/, imported as zola3d_b200."""
    if "zola3d_b200" not in sys.modules:
        d = os.path.join(ROOT, "zola-3d_b200")
        spec = importlib.util.spec_from_file_location("zola3d_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["zola3d_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["zola3d_b200"]


# ------------------------------------------------------------------ optics --
def _zernike(kind):
    """Aberrations in radians: astigmatic (15 modes), saddle point (28) or tetrapod (45)."""
    if kind == "astig":
        z = np.zeros(15)
        z[5] = 0.08 * TWO_PI
        z[[7, 8, 12]] = np.random.default_rng(11).normal(0, 0.02, 3) * TWO_PI
    elif kind == "saddle":
        z = np.zeros(28)
        z[9] = 0.3 * TWO_PI
    else:
        z = np.random.default_rng(12).normal(0, 0.02, 45) * TWO_PI
        z[:3] = 0
        z[5], z[13], z[25] = 0.6 * TWO_PI, 0.3 * TWO_PI, 0.15 * TWO_PI
    return z


_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _ctx():
    return _keep("ctx", lambda: _pkg().Context(0))


def _psf(N, kind, kz_reset=False, n_wat=1.518):
    def make():
        z = _pkg()
        zern = np.zeros(int(kind)) if kind.isdigit() else _zernike(kind)
        return z.PSF(_ctx(), z.optics(size_fft=N, sigma=0.9, kz_reset=kz_reset, n_wat=n_wat, **OPT), zern)
    return _keep(("psf", N, kind, kz_reset, n_wat), make)


def _zern_modes(nz, x, y, inside):
    """Un-normalised Zernike modes 0 .. nz - 1 (n = 0, 1, ..., m = -n, -n + 2, ..., n) on the pupil grid."""
    rho, th = np.hypot(x, y), np.arctan2(y, x)
    out, n = [], 0
    while len(out) < nz:
        for m in range(-n, n + 1, 2):
            am, s = abs(m), np.zeros_like(rho)
            for k in range((n - am) // 2 + 1):
                c = (-1) ** k * math.factorial(n - k) / (math.factorial(k) * math.factorial((n + am) // 2 - k) *
                                                         math.factorial((n - am) // 2 - k))
                s = s + c * rho ** (n - 2 * k)
            out.append(np.where((rho < 1) & inside, s * (np.cos(am * th) if m >= 0 else np.sin(am * th)), 0.0))
        n += 1
    return np.array(out[:nz])


class _Model:
    """The PSF model in 64 bits: pupil field, partial DFTs, circular Gaussian blur, normalised crop."""

    def __init__(self, N, zern, sigma=0.9, n_wat=1.518, kz_reset=False):
        c, ring = N / 2 - 0.5, (OPT["na"] / OPT["wavelength"]) ** 2
        u = (np.arange(N) - c) / (N * DX)
        rows = np.nonzero(u * u + u[N // 2] ** 2 <= ring)[0]
        self.N, self.a0, self.D, self.sigma = N, rows[0], len(rows), sigma
        u = u[rows]
        rr = u[:, None] ** 2 + u[None, :] ** 2
        inside = rr <= ring
        wat, oil = (n_wat / OPT["wavelength"]) ** 2, (OPT["n_oil"] / OPT["wavelength"]) ** 2
        dev = torch.device("cuda", 0)
        t = lambda v: torch.tensor(v, dtype=F64, device=dev)  # noqa: E731
        self.dev, self.t = dev, t
        i = np.arange(N)
        total = (((i[:, None] - c) / (N * DX)) ** 2 + ((i[None, :] - c) / (N * DX)) ** 2 <= ring).sum()
        self.pupil = t(np.where(inside, 1 / math.sqrt(total), 0.0))
        kz = TWO_PI * np.sqrt(np.abs(wat - rr))
        self.kz = t(np.where(inside & ((wat > rr) | kz_reset), kz, 0.0))
        self.isim = t(np.where(inside & (wat > rr), 1.0, 0.0))
        self.kzoil = t(np.where(inside & (oil > rr), TWO_PI * np.sqrt(np.maximum(oil - rr, 0)), 0.0))
        self.k = t(u * TWO_PI)
        radius = OPT["na"] / OPT["wavelength"] * N * DX
        x = (np.arange(self.a0, self.a0 + self.D) - c) / radius
        self.all_modes = t(_zern_modes(45, x[:, None] + 0 * x, x[None, :] + 0 * x[:, None], inside))
        self.phase = (t(zern)[:, None, None] * self.modes(len(zern))).sum(0)

    def modes(self, nz):
        return self.all_modes[:nz]

    def window(self, R, sigma=None):
        """(C, G, dG / dsigma) of an R x R region."""
        N, sigma = self.N, sigma or self.sigma
        W = 1 << (min(2 * R, N) - 1).bit_length()
        m = np.outer(np.arange(W) - W // 2, self.a0 + np.arange(self.D) + N // 2) % N
        C = torch.tensor(np.exp(2j * math.pi * m / N), dtype=C128, device=self.dev)
        f = np.fft.fftfreq(W, 1 / W)
        f[W // 2] = -W // 2
        s = W / (TWO_PI * sigma)
        g = np.exp(-0.5 * f * f / s ** 2)
        cs = np.cos(TWO_PI * (np.outer(np.arange(W), np.arange(W)) % W) / W)
        h, dh = cs @ g / W, cs @ (-g * f * f / (s * s * sigma)) / W
        d = (np.arange(R)[:, None] - R // 2 - np.arange(W)[None, :] + W // 2) % W
        return C, self.t(h[d]), self.t(dh[d])

    def maps(self, R, xyz, derivs=False, win=None):
        """psi (n, R, R), and with derivs dpsi / d(x, y, z) (n, 3, R, R)."""
        C, G, _ = win or self.window(R)
        kx, ky = self.k[:, None], self.k[None, :]
        x, y, z = (xyz[:, q, None, None] for q in range(3))
        lat = kx * x + ky * y + self.phase
        Q = torch.complex(self.pupil * torch.cos(lat + self.kz * z), self.pupil * torch.sin(lat + self.kz * z * self.isim))
        S = Q @ C.T
        E = C @ S
        out = [E.real ** 2 + E.imag ** 2]
        if derivs:
            for dE in (C @ (1j * kx * S), C @ ((1j * ky * Q) @ C.T), C @ ((1j * self.kz * Q) @ C.T)):
                out.append(2 * (E.real * dE.real + E.imag * dE.imag))
        T = G @ torch.stack(out, 1) @ G.T
        sg = torch.where(T[:, :1] < 0, -1.0, 1.0).to(F64)
        tot = T[:, :1].abs().sum((2, 3), keepdim=True)
        psi = T[:, :1].abs() / tot
        if not derivs:
            return psi[:, 0]
        dT = sg * T[:, 1:]
        return psi[:, 0], (dT - psi * dT.sum((2, 3), keepdim=True)) / tot

    def chunked(self, R, xyz, derivs=False):
        """maps() in pieces of a few GB."""
        W = 1 << (min(2 * R, self.N) - 1).bit_length()
        step, win = max(1, (1 << 31) // (16 * W * W * (5 if derivs else 2))), self.window(R)
        got = [self.maps(R, xyz[a:a + step], derivs, win) for a in range(0, len(xyz), step)]
        return tuple(torch.cat(v) for v in zip(*got)) if derivs else torch.cat(got)


def _model(N, kind, **kw):
    zern = np.zeros(int(kind)) if kind.isdigit() else _zernike(kind)
    return _keep(("model", N, kind, tuple(sorted(kw.items()))), lambda: _Model(N, zern, **kw))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


# -------------------------------------------------------------------- cases --
# The mixed job is 50% astigmatic 16 x 16, 30% saddle-point 24 x 24 and 20% tetrapod 48 x 48 regions.
MIX = [("astig", 64, 16, 0.5, 0.6, 20.0), ("saddle", 128, 24, 0.3, 1.0, 20.0), ("tetra", 128, 48, 0.2, 2.0, 30.0)]


def listed():
    return [
        # one batch of an offline job over mixed calibrations: pinned host arrays in and out
        dict(name="mixed_100k", kind="mixed", n=100000),
        # the plain localization of a movie segment: 1,000 small regions from host arrays
        dict(name="fit_1000x16", kind="fit", psf="astig", N=64, R=16, n=1000, split=True, scmos=False),
        # one camera frame's emitters, fitted as they arrive: latency and launches count
        dict(name="fit_12x24", kind="fit", psf="tetra", N=128, R=24, n=12, split=True, scmos=False),
        # a batch from an sCMOS camera, each region with its map of var / gain^2
        dict(name="fit_scmos_3001x40", kind="fit", psf="tetra", N=128, R=40, n=3001, split=True, scmos=True),
        # the FP64 form, used where every fit has to agree with the reference to rounding
        dict(name="fit_fp64_800x24", kind="fit", psf="astig", N=128, R=24, n=800, split=False, scmos=False),
        # the model and its derivatives, for simulations, residuals and precision estimates
        dict(name="model_200x32", kind="model", psf="tetra", N=128, R=32, n=200, derivs=True, split=False),
        # detection of a stack of uint16 frames against a 41-slice library
        dict(name="detect_48x256", kind="detect", psf="tetra", N=128, SX=256, SY=256, R=40, n=48, zr=2.0, step=0.1,
             u16=True),
        # detection while a camera runs: two frames of a cropped sensor, photons as doubles
        dict(name="detect_2x130", kind="detect", psf="astig", N=64, SX=130, SY=130, R=16, n=2, zr=0.6, step=0.1,
             u16=False),
        # the whole frame pipeline: uint16 frames in, localization rows out
        dict(name="localize_96x256", kind="localize", psf="tetra", N=128, S=256, R=40, n=96, zr=2.0, camera="u16",
             split=True, emitters=5),
        # calibration: likelihood and gradient of a bead stack, as an outer optimiser calls it
        dict(name="calib_grad", kind="calib", op="backward", nz=45, nb=5, ns=61, R=32, iters=0),
        # calibration: Levenberg-Marquardt iterations of the Zernike fit
        dict(name="calib_fit", kind="calib", op="fit", nz=45, nb=5, ns=61, R=32, iters=3),
        # drift of an acquisition from its localizations
        dict(name="drift_12k", kind="drift", n=12000, bins=12, L=1500.0, Lz=400.0, pixel=10.0, max_um=0.3),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["mixed", "fit", "fit", "fit", "model", "detect", "detect", "localize", "calib", "calib", "drift"])
    psf = rng.choice(["astig", "saddle", "tetra"])
    N = 64 if psf == "astig" and rng.random() < 0.6 else 128
    if kind == "mixed":
        return dict(kind=kind, n=_log(rng, 500, 90000))
    if kind == "fit":
        split = rng.random() < 0.7
        R = 2 * rng.randint(4, 24 if N == 128 else 16)
        return dict(kind=kind, psf=psf, N=N, R=R, n=_log(rng, 1, 9000 if split else 900), split=split,
                    scmos=rng.random() < 0.3)
    if kind == "model":
        return dict(kind=kind, psf=psf, N=N, R=2 * rng.randint(4, 30), n=_log(rng, 1, 1000), derivs=rng.random() < 0.6,
                    split=rng.random() < 0.3)
    if kind == "detect":
        R = 2 * rng.randint(5, 24 if N == 128 else 15)
        S = rng.randint(max(2 * R, 48), 280)
        return dict(kind=kind, psf=psf, N=N, SX=S, SY=S if rng.random() < 0.6 else rng.randint(max(2 * R, 48), S), R=R,
                    n=_log(rng, 1, 48), zr=round(rng.uniform(0.4, 2.0), 2), step=0.1, u16=rng.random() < 0.5)
    if kind == "localize":
        R = 2 * rng.randint(7, 20 if N == 128 else 15)
        return dict(kind=kind, psf=psf, N=N, S=rng.randint(96, 256), R=R, n=_log(rng, 2, 90),
                    zr=round(rng.uniform(0.5, 1.5), 2), camera=rng.choice(["u16", "photons", "scmos"]),
                    split=rng.random() < 0.7, emitters=rng.randint(1, 8))
    if kind == "calib":
        op = rng.choice(["forward", "backward", "fit"])
        return dict(kind=kind, op=op, nz=rng.choice([15, 21, 28, 36, 45]), nb=rng.randint(1, 5), ns=rng.randint(9, 61),
                    R=2 * rng.randint(8, 16), iters=rng.randint(1, 3) if op == "fit" else 0)
    return dict(kind=kind, n=_log(rng, 1000, 12000), bins=rng.randint(3, 12), L=round(rng.uniform(500, 1500), 1),
                Lz=round(rng.uniform(100, 400), 1), pixel=rng.choice([10.0, 15.0, 20.0]),
                max_um=rng.choice([0.15, 0.2, 0.3]))


# ------------------------------------------------------------------- inputs --
def _rois(psf, N, R, n, zr, bg, seed, scmos=False):
    """(rois, init, scmos map) on the device: Poisson regions around emitters of log-normal brightness, started at
    the region's centre, at the nearest depth of a 0.1 um library, with border background and summed photons."""
    g, dev = _gen(seed), "cuda"
    u = lambda a, b, *s: a + (b - a) * torch.rand(*s, generator=g, device=dev, dtype=F64)  # noqa: E731
    xyz = torch.cat([u(-DX, DX, n, 2), u(-zr, zr, n, 1)], 1)
    A = 3000 * torch.exp(0.5 * torch.randn(n, generator=g, device=dev, dtype=F64))
    var = torch.exp(0.5 * torch.randn(n, R, R, generator=g, device=dev, dtype=F64)).float() if scmos else None
    mu = A[:, None, None] * _model(N, psf).chunked(R, xyz) + bg
    rois = torch.poisson(mu + var if scmos else mu, generator=g).float()
    rim = torch.cat([rois[:, 0], rois[:, -1], rois[:, 1:-1, 0], rois[:, 1:-1, -1]], 1).double().mean(1)
    init = torch.zeros(n, 5, dtype=F64, device=dev)
    init[:, 2] = (torch.floor(xyz[:, 2] / 0.1) + 0.5) * 0.1
    init[:, 3] = (rois.double().sum((1, 2)) - rim * R * R).clamp(min=100.0)
    init[:, 4] = rim
    return rois, init, var


def _fit_prm(R, zr, split):
    z = _pkg()
    return z.PSF.fit_params(-zr - 0.3, zr + 0.3, R * DX / 2, max_iter=50, tol_xyz=1e-4,
                            precision=z.ZOLA_PREC_SPLIT if split else z.ZOLA_PREC_FP64)


def _fit_range(case):
    return {"astig": (0.6, 20.0), "saddle": (1.0, 20.0), "tetra": (1.5, 30.0)}[case["psf"]]


def _outs(n, pin=False):
    o = dict(theta=torch.zeros(n, 5, dtype=F64, pin_memory=pin), crlb=torch.zeros(n, 5, dtype=F64, pin_memory=pin),
             nll=torch.zeros(n, dtype=F64, pin_memory=pin), status=torch.zeros(n, dtype=torch.int32, pin_memory=pin),
             iters=torch.zeros(n, dtype=torch.int32, pin_memory=pin))
    return {k: v.numpy() for k, v in o.items()}


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _frames(case, seed):
    """Photon frames (n, SX, SY) on the device: Poisson emitters on a flat background."""
    SX, SY, P, n = case.get("SX", case.get("S")), case.get("SY", case.get("S")), 64 if case["N"] == 128 else 48, case["n"]
    rng = np.random.default_rng(seed)
    k = rng.poisson(case.get("emitters", 5), n)
    fr, m, bg = np.repeat(np.arange(n), k), int(k.sum()), 30.0
    cx, cy = rng.uniform(0, SX, m), rng.uniform(0, SY, m)
    zz, amp = rng.uniform(-0.9 * case["zr"], 0.9 * case["zr"], m), rng.lognormal(math.log(4000.0), 0.5, m)
    img = torch.full((n, SX + P, SY + P), bg, dtype=F64, device="cuda")
    if m:
        t = lambda v: torch.tensor(v, device="cuda")  # noqa: E731
        ix, iy = cx.astype(np.int64), cy.astype(np.int64)
        psi = _model(case["N"], case["psf"]).chunked(P, t(np.c_[(ix - cx) * DX, (iy - cy) * DX, zz]))
        for e in range(m):  # emitter by emitter: the sum's order is fixed
            img[fr[e], ix[e]:ix[e] + P, iy[e]:iy[e] + P] += amp[e] * psi[e]
    h = P // 2
    return torch.poisson(img[:, h:h + SX, h:h + SY].contiguous(), generator=_gen(seed))


OFFSET, GAIN = 100.0, 2.0  # uint16 cameras: counts = photons * gain + offset


def _u16(frames):
    return (frames * GAIN + OFFSET).clamp(max=65535).cpu().numpy().astype(np.uint16)


def _detector(case):
    S = (case.get("SX", case.get("S")), case.get("SY", case.get("S")))
    step = case.get("step", 0.1)
    key = ("det", case["psf"], case["N"], S, case["R"], case["zr"], step)
    return _keep(key, lambda: _pkg().Detector(_psf(case["N"], case["psf"], kz_reset=True), S[0], S[1], case["R"],
                                              -case["zr"], case["zr"], step, 0.1))


def _poly(c, R):
    i = torch.arange(R, dtype=F64, device=c.device)
    a, b = i[:, None] + 0 * i, i[None, :] + 0 * i[:, None]
    return torch.einsum("...k,kxy->...xy", c, torch.stack([1 + 0 * a, a, a * a, b, a * b, b * b]))


def _beads(case, seed):
    """(stacks, dz, photons, zernike start, bead parameters) of a bead calibration, 1.33 sample, Poisson noise."""
    nz, nb, ns, R = case["nz"], case["nb"], case["ns"], case["R"]
    rng = np.random.default_rng(seed)
    zern = rng.normal(0, 0.05, nz) * TWO_PI
    zern[:3] = 0
    zern[5] += 0.1 * TWO_PI
    dz = (np.arange(ns) - ns // 2) * 3.0 / ns
    xyz = rng.uniform(-0.05, 0.05, (nb, 3))
    photons = np.full((nb, ns), 20000.0) * (1 + 0.1 * np.cos(dz / 0.6))
    t = lambda v: torch.tensor(v, dtype=F64, device="cuda")  # noqa: E731
    M = _model(128, str(nz), n_wat=1.33)
    mu = _bead_mean(M, R, t(zern), 1.0, t(xyz), t(dz), t(photons), t(np.tile([50.0, 0, 0, 0, 0, 0], (nb, 1))))
    stacks = torch.poisson(mu, generator=_gen(seed)).cpu().numpy()
    bead = np.zeros((nb, 3 + ns + 6))
    bead[:, 3 + ns] = 50.0
    start = np.zeros(nz)
    start[5] = 0.08 * TWO_PI
    return stacks, dz, photons, start, bead


def _localizations(case, seed):
    """A static structure localized over 5,000 frames while the stage drifts (nm)."""
    rng = np.random.default_rng(seed)
    pts = np.c_[rng.uniform(0, case["L"], (150, 2)), rng.uniform(0, case["Lz"], 150)]
    fr = rng.integers(0, 5000, case["n"])
    vel = np.array([0.01, -0.008, 0.004])
    xyz = pts[rng.integers(0, 150, case["n"])] + np.outer(fr, vel) + rng.normal(0, 4.0, (case["n"], 3))
    return xyz, fr.astype(np.int32), np.full((case["n"], 3), 4.0)


def prepare(case, seed):
    z, kind, st = _pkg(), case["kind"], {"case": case}
    if kind == "mixed":
        st["classes"] = []
        for c, (psf, N, R, frac, zr, bg) in enumerate(MIX):
            n = max(1, round(case["n"] * frac))
            rois, init, _ = _rois(psf, N, R, n, zr, bg, 10 * seed + c)
            st["classes"].append(dict(psf=_psf(N, psf), rois=_pinned(rois), init=_pinned(init),
                                      prm=_fit_prm(R, zr, True), out=_outs(n, pin=True)))
    elif kind == "fit":
        zr, bg = _fit_range(case)
        rois, init, var = _rois(case["psf"], case["N"], case["R"], case["n"], zr, bg, seed, case["scmos"])
        st.update(psf=_psf(case["N"], case["psf"]), rois=rois.cpu().numpy(), init=init.cpu().numpy(),
                  scmos=var.cpu().numpy() if case["scmos"] else None, prm=_fit_prm(case["R"], zr, case["split"]))
    elif kind == "model":
        rng = np.random.default_rng(seed)
        st.update(psf=_psf(case["N"], case["psf"]), xyz=rng.uniform(-1, 1, (case["n"], 3)) * [0.3, 0.3, 1.0])
    elif kind == "detect":
        f = _frames(case, seed)
        st.update(det=_detector(case), frames=_u16(f) if case["u16"] else f.cpu().numpy())
    elif kind == "localize":
        f = _frames(case, seed)
        st.update(det=_detector(case), psf=_psf(case["N"], case["psf"]))
        if case["camera"] == "u16":
            st["frames"] = _u16(f)
        elif case["camera"] == "photons":
            st["frames"] = f.cpu().numpy()
        else:
            rng, S = np.random.default_rng(seed), (case["S"], case["S"])
            off, gain = rng.normal(100, 1, S), rng.normal(2.0, 0.05, S)
            st["maps"] = (off, gain, rng.lognormal(math.log(4.0), 0.3, S))
            noise = rng.normal(0, 1, (case["n"],) + S) * np.sqrt(st["maps"][2])
            st["frames"] = (f.cpu().numpy() * gain + off + noise).astype(np.float32)
    elif kind == "calib":
        stacks, dz, photons, start, bead = _beads(case, seed)
        st.update(cal=z.Calibration(_psf(128, str(case["nz"]), n_wat=1.33), stacks, dz, photons=photons), start=start,
                  bead=bead)
    else:
        st["locs"] = _localizations(case, seed)
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------- run --
BEST = 256  # candidates asked for per frame, best first


def _block(rows):
    """Lists of candidate rows as one array (frames, BEST, 7); a shorter list ends in zeros."""
    out = np.zeros((len(rows), BEST, 7))
    for f, r in enumerate(rows):
        out[f, :len(r)] = r
    return out


def run(st):
    z, case = _pkg(), st["case"]
    kind = case["kind"]
    if kind == "mixed":
        z.fit_mixed(_ctx(), st["classes"])
        return [c["out"] for c in st["classes"]]
    if kind == "fit":
        return st["psf"].fit(st["rois"], st["init"], st["prm"], scmos=st["scmos"])
    if kind == "model":
        return st["psf"].model(case["R"], st["xyz"], derivs=case["derivs"],
                               precision=z.ZOLA_PREC_SPLIT if case["split"] else z.ZOLA_PREC_FP64)
    if kind == "detect":
        if case["u16"]:
            rows, counts = st["det"].detect_u16(st["frames"], adu=1.0, gain=GAIN, offset=OFFSET, cap=BEST)
        else:
            rows, counts = st["det"].detect(st["frames"], cap=BEST)
        return _block(rows), counts
    if kind == "localize":
        args = dict(minZ=-case["zr"], maxZ=case["zr"], max_iter=50,
                    precision=z.ZOLA_PREC_SPLIT if case["split"] else z.ZOLA_PREC_FP64)
        if case["camera"] == "u16":
            rows = z.localize_frames_u16(_ctx(), st["det"], st["psf"], st["frames"], adu=1.0, gain=GAIN, offset=OFFSET,
                                         **args)
        elif case["camera"] == "photons":
            rows = z.localize_frames(_ctx(), st["det"], st["psf"], st["frames"], **args)
        else:
            rows = z.localize_frames_scmos(_ctx(), st["det"], st["psf"], st["frames"], *st["maps"], **args)
        out = np.zeros(64 * case["n"], rows.dtype)  # a fixed length for every movie of this size
        out[:len(rows)] = rows
        return {c: out[c] for c in z.LOC_COLUMNS} | {"rows": len(rows)}
    if kind == "calib":
        if case["op"] == "fit":
            return st["cal"].fit(st["start"], 0.9, st["bead"], max_iter=case["iters"])
        return (st["cal"].backward if case["op"] == "backward" else st["cal"].forward)(st["start"], 0.9, st["bead"])
    return z.drift(_ctx(), *st["locs"], pixel_nm=case["pixel"], bins=case["bins"], max_drift_um=case["max_um"])


# --------------------------------------------------------------------- work --
def _eval_flops(N, R, derivs):
    """One model by partial DFTs over the D x D pupil square and the W x W window, complex multiply-add = 8."""
    D, W = (30 if N == 64 else 60), 1 << (min(2 * R, N) - 1).bit_length()
    dft = 8 * W * D * D, 8 * W * W * D
    blur = 2 * R * W * W + 2 * R * R * W
    return 3 * dft[0] + 4 * dft[1] + 4 * blur if derivs else dft[0] + dft[1] + blur


def work(case):
    kind = case["kind"]
    if kind == "mixed":
        w = [work(dict(kind="fit", N=N, R=R, n=max(1, round(case["n"] * f)), scmos=False)) for _, N, R, f, _, _ in MIX]
        return {k: sum(x[k] for x in w) for k in w[0]}
    if kind == "fit":  # about seven evaluations a fit
        n, RR = case["n"], case["R"] ** 2
        return {"bytes": n * (RR * (8 if case["scmos"] else 4) + 40 + 96), "flops": 7 * n * _eval_flops(case["N"], case["R"], True)}
    if kind == "model":
        n, maps = case["n"], 4 if case["derivs"] else 1
        return {"bytes": n * (24 + 8 * maps * case["R"] ** 2), "flops": n * _eval_flops(case["N"], case["R"], case["derivs"])}
    if kind in ("detect", "localize"):  # correlation with every library slice through real FFTs, then the peaks
        SX, SY = case.get("SX", case.get("S")), case.get("SY", case.get("S"))
        Z, M = math.ceil(2 * case["zr"] / case.get("step", 0.1)), (SX + case["R"] / 2) * (SY + case["R"] / 2)
        flops = case["n"] * (2.5 * M * math.log2(M) * (Z + 1) + Z * (6 * M + 20 * SX * SY))
        w = {"bytes": case["n"] * SX * SY * (2 if case.get("u16", case.get("camera") == "u16") else 8), "flops": flops}
        if kind == "localize":  # ten fits a frame
            f = work(dict(kind="fit", N=case["N"], R=case["R"], n=10 * case["n"], scmos=case["camera"] == "scmos"))
            w = {k: w[k] + f[k] for k in w}
        return w
    if kind == "calib":
        items, RR = case["nb"] * case["ns"], case["R"] ** 2
        fwd = _eval_flops(128, case["R"], False)
        evals = 1 if case["op"] == "forward" else 3
        flops = items * fwd * evals
        if case["op"] == "fit":
            ndir = case["nz"] - 3 + 1 + 3
            flops = (case["iters"] + 1) * items * (2 * 3 * fwd + ndir * fwd + RR * (ndir + 7) ** 2)
        return {"bytes": items * RR * 8 + 60 * 60 * 8 * case["nz"], "flops": flops}
    size = 2 ** math.ceil(math.log2(case["max_um"] * 1000 / case["pixel"]))
    ext = [math.ceil(v / case["pixel"]) for v in (case["L"], case["L"], case["Lz"])]
    win = math.prod(max(1, math.ceil((e - size / 2) / (size / 2))) for e in ext)
    P, pairs = 8 * math.prod(min(size, 1 << (e - 1).bit_length()) for e in ext), case["bins"] * (case["bins"] - 1) // 2
    return {"bytes": case["n"] * 52, "flops": win * (case["bins"] + pairs) * 2.5 * P * math.log2(P)}


# -------------------------------------------------------------------- exact --
class _Lm:
    """The damped Gauss-Newton fit of (x, y, z, A, B) to Poisson regions, for all regions at once in 64 bits."""

    FLOOR = (1.0, 1.0, 1.0, 1e-10, 1e-6)

    def __init__(self, M, rois, init, var, zr, R):
        self.M, self.R, self.win, self.d, self.v = M, R, M.window(R), rois, var
        self.lo = torch.tensor([-R * DX / 2, -R * DX / 2, -zr - 0.3, 1.0, 0.01], dtype=F64, device="cuda")
        self.hi = torch.tensor([R * DX / 2, R * DX / 2, zr + 0.3, math.inf, math.inf], dtype=F64, device="cuda")
        self.floor = torch.tensor(self.FLOOR, dtype=F64, device="cuda")
        self.th = self.clamp(init)

    def clamp(self, t):
        return torch.minimum(torch.maximum(t, self.lo), self.hi)

    def evaluate(self, idx, th):
        W = self.win[0].shape[0]
        step = max(1, (1 << 31) // (16 * W * W * 6))
        got = [self._evaluate(idx[a:a + step], th[a:a + step]) for a in range(0, len(idx), step)]
        return [torch.cat(v) for v in zip(*got)]

    def _evaluate(self, idx, th):
        psi, dpsi = self.M.maps(self.R, th, True, self.win)
        d = self.d[idx].double()
        A, B = th[:, 3, None, None], th[:, 4, None, None]
        mu = A * psi + B + (self.v[idx].double() if self.v is not None else 0.0)
        J = torch.cat([A[:, None] * dpsi, psi[:, None], torch.ones_like(psi)[:, None]], 1).flatten(2)
        bad = ~(mu > 0)
        mu1 = torch.where(bad, 1.0, mu)
        nll = torch.where(d > 0, mu1 - d - d * torch.log(mu1 / torch.where(d > 0, d, 1.0)), mu1).sum((1, 2))
        nll = torch.where(bad.any(2).any(1), math.inf, nll)
        w = lambda x: (J * x.flatten(1)[:, None]) @ J.transpose(1, 2)  # noqa: E731
        g = ((1 - d / mu1).flatten(1)[:, None] * J).sum(2)
        return nll, g, w(d / mu1 ** 2), w(1 / mu1)

    def solve(self, H, g, lam):
        L, info = torch.linalg.cholesky_ex(H + torch.diag_embed(lam[:, None] * torch.maximum(H.diagonal(dim1=1, dim2=2), self.floor)))
        ok = (info == 0) & torch.isfinite(L).all(2).all(1)
        L = torch.where(ok[:, None, None], L, torch.eye(5, dtype=F64, device=L.device))
        return torch.cholesky_solve(-g[:, :, None], L)[:, :, 0], ok

    def optimum(self, th, H, g):
        s, ok = self.solve(H, g, torch.zeros(len(th), dtype=F64, device="cuda"))
        return ok & (s[:, :3].abs().amax(1) < 1e-4) & (s[:, 3].abs() < 1e-4 * th[:, 3]) & \
            (s[:, 4].abs() < 1e-4 * th[:, 4].clamp(min=1.0))

    def fit(self):
        n, cap = len(self.th), torch.tensor([DX, DX, 2 * DX], dtype=F64, device="cuda")
        every = torch.arange(n, device="cuda")
        nll, g, H, F = self.evaluate(every, self.th)
        lam = torch.full((n,), 1e-3, dtype=F64, device="cuda")
        run = torch.isfinite(nll) & ~self.optimum(self.th, H, g)
        for _ in range(49):
            for _ in range(12):  # raise the damping where the damped matrix is not positive definite
                s, ok = self.solve(H, g, lam)
                lam = torch.where(run & ~ok, lam * 10, lam)
                if bool((ok | ~run).all()):
                    break
            run = run & ok & (lam <= 1e7)
            i = every[run]
            if not len(i):
                break
            s = s[i]
            sxy = s[:, :2].abs().amax(1)
            k = torch.where(sxy > cap[0], cap[0] / sxy, 1.0)
            k = torch.where(s[:, 2].abs() * k > cap[2], cap[2] / s[:, 2].abs(), k)
            t = self.clamp(self.th[i] + k[:, None] * s)
            f2, g2, H2, F2 = self.evaluate(i, t)
            up = f2 <= nll[i]
            a = i[up]
            self.th[a], nll[a], g[a], H[a], F[a] = t[up], f2[up], g2[up], H2[up], F2[up]
            lam[i] = torch.where(up, (lam[i] * 0.1).clamp(min=1e-7), lam[i] * 10)
            done = self.optimum(self.th[i], H[i], g[i]) & up
            run[i] = ~done & (lam[i] <= 1e7)
        crlb = torch.linalg.inv(F).diagonal(dim1=1, dim2=2).sqrt()
        return dict(theta=self.th, crlb=crlb, nll=nll, status=None, iters=None)


def _fit_exact(psf, N, R, n, zr, bg, seed, scmos):
    rois, init, var = _rois(psf, N, R, n, zr, bg, seed, scmos)
    out = _Lm(_model(N, psf), rois, init, var, zr, R).fit()
    if psf == "saddle":  # I(-z) = I(z): the Fisher matrix is singular at z = 0, and its inverse has no value there
        out["crlb"] = None
    return out


def _bead_mean(M, R, zern, sigma, xyz, dz, photons, poly, win=None):
    """Mean photons (nb, ns, R, R) of the bead stacks; phase from modes 3 and up, at depth 0 in the sample."""
    C, G, _ = win or M.window(R, sigma)
    ph = (zern[3:, None, None] * M.modes(len(zern))[3:]).sum(0) + xyz[:, None, 0, None, None] * M.k[:, None] + \
        xyz[:, None, 1, None, None] * M.k[None, :] - M.kzoil * (dz[None, :] + xyz[:, 2, None])[:, :, None, None]
    E = C @ torch.polar(M.pupil.expand_as(ph), ph) @ C.T
    T = G @ (E.real ** 2 + E.imag ** 2) @ G.T
    return T.abs() / T.abs().sum((2, 3), keepdim=True) * photons[:, :, None, None] + _poly(poly, R)[:, None]


class _Calib:
    """Likelihood, gradient and Levenberg-Marquardt fit of a bead calibration in 64 bits."""

    def __init__(self, case, seed):
        stacks, dz, photons, self.z0, self.b0 = _beads(case, seed)
        t = lambda v: torch.tensor(v, dtype=F64, device="cuda")  # noqa: E731
        self.case, self.M, self.t = case, _model(128, str(case["nz"]), n_wat=1.33), t
        self.d, self.dz, self.ph = t(stacks), t(dz), t(photons)

    def value(self, z, sigma, b, grad):
        case, R, ns = self.case, self.case["R"], self.case["ns"]
        z, b, s = self.t(z).requires_grad_(grad), self.t(b).requires_grad_(grad), self.t(sigma).requires_grad_(grad)
        C, G, dG = self.M.window(R, float(sigma))
        G = G + dG * (s - s.detach())
        mu = _bead_mean(self.M, R, z, None, b[:, :3], self.dz, self.ph + b[:, 3:3 + ns], b[:, 3 + ns:], (C, G, dG))
        mu = torch.where(mu <= 0, 1e-8, mu)
        nll = (mu - self.d * torch.log(mu)).sum()
        if not grad:
            return np.float64(nll.item())
        gz, gs, gb = torch.autograd.grad(nll, (z, s, b))
        gz[:3] = 0
        return np.float64(nll.item()), gz.cpu().numpy(), np.float64(gs.item()), gb.cpu().numpy(), mu.detach()

    def jacobian(self, z, sigma, b):
        """d mu / d theta, (pixels, parameters) in the order modes 3 .., sigma, bead parameters."""
        case, M = self.case, self.M
        nz, nb, ns, R = case["nz"], case["nb"], case["ns"], case["R"]
        C, G, dG = M.window(R, float(sigma))
        z, b = self.t(z), self.t(b)
        pb, off = 3 + ns + 6, nz - 2
        J = torch.zeros(nb, ns, R, R, off + nb * pb, dtype=F64, device="cuda")
        modes = M.modes(nz)[3:]
        poly = _poly(torch.eye(6, dtype=F64, device="cuda"), R)
        for k in range(nb):
            ph = (z[3:, None, None] * modes).sum(0) + b[k, 0] * M.k[:, None] + b[k, 1] * M.k[None, :] - \
                M.kzoil * (self.dz + b[k, 2])[:, None, None]
            Q = torch.polar(M.pupil.expand_as(ph), ph)
            E = C @ Q @ C.T
            I = E.real ** 2 + E.imag ** 2  # noqa: E741
            T = G @ I @ G.T
            sg, tot = torch.where(T < 0, -1.0, 1.0).to(F64), T.abs().sum((1, 2), keepdim=True)
            psi, A = T.abs() / tot, (self.ph[k] + b[k, 3:3 + ns])[:, None, None]

            def push(dT):
                dT = sg * dT
                return A * (dT - psi * dT.sum((1, 2), keepdim=True)) / tot

            def phase(p):
                dE = C @ (1j * Q * p) @ C.T
                return push(G @ (2 * (E.real * dE.real + E.imag * dE.imag)) @ G.T)

            for m in range(nz - 3):
                J[k, ..., m] = phase(modes[m])
            J[k, ..., nz - 3] = push(dG @ I @ G.T + G @ I @ dG.T)
            o = off + k * pb
            own = torch.where(M.pupil > 0, 1.0, 0.0)
            for q, p in enumerate((own * M.k[:, None], own * M.k[None, :], -own * M.kzoil)):
                J[k, ..., o + q] = phase(p)
            for s in range(ns):
                J[k, s, :, :, o + 3 + s] = psi[s]
            J[k, ..., o + 3 + ns:o + pb] = poly.permute(1, 2, 0)
        return J.flatten(0, 3)

    def fit(self):
        case = self.case
        nz, nb, pb = case["nz"], case["nb"], 3 + case["ns"] + 6
        th = np.concatenate([self.z0[3:], [0.9], self.b0.ravel()])

        def split(t):
            return np.concatenate([self.z0[:3], t[:nz - 3]]), t[nz - 3], t[nz - 2:].reshape(nb, pb)

        def both(t):
            f, gz, gs, gb, mu = self.value(*split(t), True)
            w = torch.where(mu > 1e-8, 1 / mu, 0.0).flatten()
            J = self.jacobian(*split(t))
            return f, np.concatenate([gz[3:], [gs], gb.ravel()]), (J * w[:, None]).T @ J

        f, g, H = both(th)
        lam, it = 1e-3, 0
        while it < case["iters"]:
            A = H + torch.diag(lam * H.diagonal().clamp(min=1e-12))
            L, info = torch.linalg.cholesky_ex(A)
            if int(info):
                lam *= 10
                it += 1
                continue
            t2 = th + torch.cholesky_solve(-self.t(g)[:, None], L)[:, 0].cpu().numpy()
            t2[nz - 3] = max(t2[nz - 3], 0.05)
            a = t2[nz - 2:].reshape(nb, pb)[:, 3:-6]
            np.maximum(a, 1 - self.ph.cpu().numpy(), out=a)
            f2 = self.value(*split(t2), False)
            it += 1
            if f2 <= f:
                small = f - f2 < 1e-9 * max(1.0, abs(f))
                th, lam = t2, max(lam * 0.1, 1e-9)
                f, g, H = both(th)
                if small:
                    break
            else:
                lam *= 10
        return [*split(th), f, None]


def _scores(case, frames):
    """Correlation scores (n, Z, SX, SY) of photon frames with the zero-mean library, and the library's depths."""
    SX, SY, R, step = case["SX"], case["SY"], case["R"], case["step"]
    Z, h = math.ceil(2 * case["zr"] / step), R // 2
    zs, z = [], -case["zr"]
    for _ in range(Z):
        zs.append(z)
        z += step
    M = _model(case["N"], case["psf"], kz_reset=True)
    xyz = torch.zeros(Z, 3, dtype=F64, device="cuda")
    xyz[:, 2] = torch.tensor(zs)
    lib = M.chunked(R, xyz)
    lib = lib - lib.mean((1, 2), keepdim=True)
    vp = (lib ** 2).mean((1, 2))
    i, j = np.arange(SX)[:, None], np.arange(SY)[None, :]
    v1, v2 = np.where(i < h - 1, i + 1, h), np.where(i > SX - h - 2, SY - i - 1, h)
    w1, w2 = np.where(j < h - 1, j + 1, h), np.where(j > SX - h - 2, SY - j - 2, h)
    norm = torch.tensor(((v1 + v2) * (w1 + w2)).astype(float), device="cuda")
    P = [1 << (s + R - 1).bit_length() for s in (SX, SY)]
    K = torch.fft.rfft2(torch.roll(torch.nn.functional.pad(lib, (0, P[1] - R, 0, P[0] - R)), (-h, -h), (1, 2))).conj()
    scale = 1 / math.sqrt((1 << (2 * SX - 1).bit_length()) * (1 << (2 * SY - 1).bit_length()))

    def box(x):  # sums over [i - h + 1, i + h] of both axes
        for d in (1, 2):
            x = torch.nn.functional.pad(x, (h - 1, h) if d == 2 else (0, 0, h - 1, h)).unfold(d, 2 * h, 1).sum(-1)
        return x

    for f in frames.split(max(1, (1 << 31) // (16 * P[0] * P[1] * (Z + 1)))):
        r = f.float().double()
        a, b = box(r) / norm, box(r * r) / norm
        var = (b - a * a)[:, None]
        corr = torch.fft.irfft2(torch.fft.rfft2(f, s=P)[:, None] * K, s=P)[:, :, :SX, :SY]
        s = torch.sqrt(vp[None, :, None, None] * var)
        yield torch.where(s > 0, corr * scale / s, -2.0)


def _peak_rows(case, sc):
    """The candidate rows of one frame's scores, best first."""
    Z, SX, SY = sc.shape
    lo = max(3, case["R"] // 2)
    inner = torch.zeros(SX, SY, dtype=torch.bool, device=sc.device)
    inner[lo:SX - lo, lo:SY - lo] = True
    pad = torch.nn.functional.pad
    tmp, rows = torch.zeros(SX, SY, dtype=F64, device=sc.device), []
    for r in range(Z):
        s = sc[r]
        tmp = torch.where(inner & (s > 0), pad(s, (3, 3), value=-math.inf).unfold(1, 7, 1).amax(-1), tmp)
        col = pad(tmp.T, (3, 3), value=-math.inf).unfold(1, 7, 1).amax(-1).T
        j, i = torch.nonzero((inner & (s > 0.1) & (s == tmp) & (s == col)).T, as_tuple=True)

        def top(a, c, w, ok):
            v = s[i, j]
            p = (c - a) / (2 * w), (c + a - 2 * v) / (2 * w * w)
            return torch.where(ok, -p[0] / (2 * p[1]), 0.0)

        tz = top(sc[max(r - 1, 0)][i, j], sc[min(r + 1, Z - 1)][i, j], case["step"],
                 torch.full_like(i, 1 < r < Z - 1, dtype=torch.bool))
        tx = top(s[i - 1, j], s[i + 1, j], DX, (i > 1) & (i < SX - 1))
        ty = top(s[i, j - 1], s[i, j + 1], DX, (j > 1) & (j < SY - 1))
        rows.append(torch.stack([s[i, j], torch.full_like(tz, r), i.double(), j.double(), tz, tx, ty], 1))
    rows = torch.cat(rows)
    return rows[torch.sort(rows[:, 0], descending=True, stable=True)[1]]


def _detect_exact(case, seed):
    f = _frames(case, seed)
    if case["u16"]:
        counts = torch.tensor(_u16(f).astype(np.float64), device="cuda")
        f = (counts * (1.0 / GAIN) + (-OFFSET * 1.0 / GAIN)).clamp(min=0)
    rows = [_peak_rows(case, s) for part in _scores(case, f) for s in part]
    return [_block([r[:BEST].cpu().numpy() for r in rows]), np.array([len(r) for r in rows], np.int32)]


def _drift_peak(im):
    """Centroid, relative to the centre, of the values above the 95% quantile around the first maximum."""
    S, at = im.shape, np.unravel_index(int(im.argmax()), im.shape)
    half = [max(1, min(11, n - 1) - 1 + min(11, n - 1) % 2) // 2 for n in S]  # odd boxes of at most 11 voxels
    box = tuple(slice(max(0, a - h), min(n, a + h + 1)) for a, h, n in zip(at, half, S))
    p = im[box]
    thr = np.sort(p.ravel())[int((p.size - 1) * .95)]
    w = np.where(p > thr, p, 0.0)
    ix = np.meshgrid(*[np.arange(b.start, b.stop) for b in box], indexing="ij")
    return [-((w * x).sum() / w.sum() - n // 2) for x, n in zip(ix, S)]


def _drift_exact(case, seed):
    """Bin drifts and per-localization drifts with 64-bit transforms (the library's are 32-bit)."""
    xyz, fr, crlb = _localizations(case, seed)
    bins, px = case["bins"], case["pixel"]
    size = 2 ** math.ceil(math.log2(case["max_um"] * 1000 / px))
    mn, mx = xyz.min(0), np.maximum(xyz.max(0), 4.9e-324)
    ext = np.maximum(np.ceil((mx - mn) / px), 1).astype(int)
    sF = [max(min(size, e), 2 ** math.ceil(math.log2(min(size, e)))) for e in ext]
    nw = [1 if s < 2 else math.ceil((e - s // 2) / (s // 2)) for s, e in zip(sF, ext)]
    prec = crlb.mean(0)
    sig = 3 * prec.max() / px
    S, P = sF[::-1], [2 * s for s in sF[::-1]]
    gauss = 1
    for d in range(3):
        f = np.fft.fftfreq(P[d], 1 / P[d])
        f[P[d] // 2] = -P[d] // 2
        g = np.exp(-.5 * f * f / (P[d] / (sig * TWO_PI)) ** 2)
        gauss = gauss * g.reshape([-1 if k == d else 1 for k in range(3)])
    gauss = torch.tensor(gauss.astype(np.float32).astype(float), device="cuda")
    rel, mf, xf = xyz - mn, int(fr.min()), int(fr.max())
    b_of = (bins * (fr.astype(np.int64) - mf)) // (1 + xf - mf)
    pairs = [(t, s) for t in range(bins - 1) for s in range(t + 1, bins)]
    t_, s_ = (torch.tensor(v, device="cuda") for v in zip(*pairs))
    res = torch.zeros(len(pairs), *S, dtype=F64, device="cuda")
    for u in np.ndindex(*nw):
        g0 = np.array([(u[d] // 2) * sF[d] * px + (u[d] % 2) * (sF[d] // 2) * px for d in range(3)])
        ok = ((rel >= g0) & (rel < g0 + np.array(sF) * px)).all(1)
        v = [np.clip(np.fmod(rel[ok, d], sF[d] * px) // px, 0, sF[d] - 1).astype(int) + sF[d] // 2 for d in range(3)]
        cube = np.zeros([bins] + P)
        np.add.at(cube, (b_of[ok], v[2], v[1], v[0]), 1.0)
        F = torch.fft.fftn(torch.tensor(cube, device="cuda"), dim=(1, 2, 3)) * gauss
        for a in range(0, len(pairs), 16):
            c = torch.fft.ifftn(F[t_[a:a + 16]] * F[s_[a:a + 16]].conj(), dim=(1, 2, 3), norm="forward").real
            c = torch.roll(c, [p // 2 for p in P], (1, 2, 3))
            res[a:a + 16] += c[:, S[0] // 2:S[0] // 2 + S[0], S[1] // 2:S[1] // 2 + S[1], S[2] // 2:S[2] // 2 + S[2]]
    pd = np.array([_drift_peak(r.cpu().numpy())[::-1] for r in res]) * px  # x, y, z
    fpb = (xf - mf) / bins
    di = np.array([mf + fpb / 2] + [s / bins * (1.0 + xf - mf) + mf + fpb / 2 for s in range(1, bins)])
    dr = np.zeros((bins, 3))
    dr[1:] = pd[:bins - 1]
    A = np.zeros((len(pairs), bins - 1))
    for k, (t, s) in enumerate(pairs):
        A[k, s - 1] = 1
        if t:
            A[k, t - 1] = -1
    if bins > 2 and len(pairs) > bins:
        for d in range(3):
            gone = []  # positions in the list that was solved, as the reference's removal counts them
            for _ in range(2):
                k = [i for i in range(len(pairs)) if i not in gone]
                if len(k) < bins - 1:
                    continue
                N = A[k].T @ A[k]
                if np.linalg.matrix_rank(N) < bins - 1:
                    continue
                sol = np.linalg.solve(N, A[k].T @ pd[k, d])
                gone += list(np.nonzero(np.abs(A[k] @ sol - pd[k, d]) > prec[d])[0])
                dr[1:, d] = sol
    out = np.zeros((len(fr), 3))
    for d in range(3):
        out[:, d] = _spline(di, dr[:, d], fr.astype(float))
    return [np.c_[di, dr], out, None]


def _spline(x, y, X):
    """Cubics through four consecutive knots, straight lines outside the knots; fewer than four knots: one polynomial."""
    L = len(x)
    if L < 4:
        return np.polynomial.Polynomial.fit(x, y, L - 1)(X)
    cub = [np.polynomial.Polynomial.fit(x[k:k + 4], y[k:k + 4], 3) for k in range(L - 3)]
    i = np.minimum(np.searchsorted(x, X, side="right"), L - 1)
    i = np.where(i == 1, 2, i)
    i = np.where(i == L - 1, L - 2, i)
    out = np.zeros_like(X)
    for k in range(L - 3):
        out = np.where(np.clip(i - 2, 0, L - 4) == k, cub[k](X), out)
    out = np.where(i == 0, cub[0].deriv()(x[0]) * (X - x[0]) + y[0], out)
    return np.where(X > x[-1], cub[-1].deriv()(x[-1]) * (X - x[-1]) + y[-1], out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mixed":
        return [_fit_exact(p, N, R, max(1, round(case["n"] * f)), zr, bg, 10 * seed + c, False)
                for c, (p, N, R, f, zr, bg) in enumerate(MIX)]
    if kind == "fit":
        return _fit_exact(case["psf"], case["N"], case["R"], case["n"], *_fit_range(case), seed, case["scmos"])
    if kind == "model":
        rng = np.random.default_rng(seed)
        xyz = torch.tensor(rng.uniform(-1, 1, (case["n"], 3)) * [0.3, 0.3, 1.0], device="cuda")
        return _model(case["N"], case["psf"]).chunked(case["R"], xyz, case["derivs"])
    if kind == "detect":
        return _detect_exact(case, seed)
    if kind == "calib":
        c = _Calib(case, seed)
        if case["op"] == "fit":
            return c.fit()
        if case["op"] == "forward":
            return c.value(c.z0, 0.9, c.b0, False)
        return list(c.value(c.z0, 0.9, c.b0, True)[:4])
    if kind == "drift":
        return _drift_exact(case, seed)
    return None  # localize: thousands of sequential candidate fits, minutes in plain numpy
