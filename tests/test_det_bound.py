"""The detection's error bound and open ranks (csrc/det_bound.h), compiled by the host compiler."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zola-3d_b200", "csrc")


@pytest.fixture(scope="module")
def bound(tmp_path_factory):
    d = tmp_path_factory.mktemp("det_bound")
    src, lib = d / "b.cpp", d / "b.so"
    src.write_text("""#include "det_bound.h"
extern "C" double pair_ratio(const double* v, int Z) { return zola::det_pair_ratio(v, Z); }
extern "C" void fft_bound(int SX, int SY, int R, int MX, int MY, double m, double p, double* kb) {
    zola::det_fft_bound(SX, SY, R, MX, MY, m, p, kb, kb + 1);
}
extern "C" int tie(double s, double next, double e) { return zola::det_tie(s, next, e); }
""")
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I", CSRC, "-o", str(lib), str(src)])
    b = ctypes.CDLL(str(lib))
    b.pair_ratio.restype = ctypes.c_double
    b.fft_bound.argtypes = [ctypes.c_int] * 5 + [ctypes.c_double] * 2 + [ctypes.c_void_p]
    b.tie.argtypes = [ctypes.c_double] * 3
    return b


@pytest.mark.parametrize("ratio", [1.0, 30.0, 1e8])
def test_bound_covers_the_partner_of_a_weak_slice(bound, ratio):
    """Two slices in one complex transform, one `ratio` times the other: the weak one's scores at 40 pixels, against
    exact rational sums, are within the bound; at 1e8 they are not within that of a slice by itself."""
    S, R, M = 48, 16, 64
    rng = np.random.default_rng(3)
    img = rng.poisson(20.0, (S, S)).astype(float)
    img[10, 11] = 4000.0
    p = rng.normal(size=(2, R, R))
    p -= p.mean((1, 2), keepdims=True)
    p[1] *= ratio * math.sqrt((p[0] ** 2).mean() / (p[1] ** 2).mean())
    var = np.ascontiguousarray((p ** 2).mean((1, 2)))
    inv_m = 1.0 / 128
    pair = bound.pair_ratio(var.ctypes.data_as(ctypes.c_void_p), 2)
    assert pair == pytest.approx(math.sqrt(1 + ratio ** 2), rel=1e-6)
    K = np.zeros((M, M), complex)
    h = R // 2
    for u in range(R):
        for v in range(R):
            K[(u - h) % M, (v - h) % M] = p[0, u, v] - 1j * p[1, u, v]
    field = np.zeros((M, M))
    field[:S, :S] = img
    corr = np.fft.ifft2(np.fft.fft2(field) * np.conj(np.fft.fft2(K))).real
    kb = {}
    for q in (1.0, pair):
        a = np.zeros(2)
        bound.fft_bound(S, S, R, M, M, inv_m, q, a.ctypes.data_as(ctypes.c_void_p))
        kb[q] = a
    worst = 0.0
    for i, j in rng.integers(h, S - h, (40, 2)):
        patch = img[i - h:i + h, j - h:j + h]
        exact = sum(Fraction(int(a)) * Fraction(float(b)) for a, b in zip(patch.ravel(), p[0].ravel()))
        vi = img[i - h + 1:i + h + 1, j - h + 1:j + h + 1].var()
        err = abs(float(Fraction(float(corr[i, j])) - exact)) * inv_m / math.sqrt(var[0] * vi)
        eps = {q: a[0] * img.max() / math.sqrt(vi) + a[1] for q, a in kb.items()}
        assert err <= eps[pair]
        worst = max(worst, err / eps[1.0])
    assert worst > 1 or ratio < 1e8


def test_pair_ratio_ignores_empty_slices(bound):
    for v, want in (([1.0], 1.0), ([1.0, 0.0], 1.0), ([4.0, 1.0, 1.0], math.sqrt(5)), ([1.0, 1.0, 9.0, 0.25], math.sqrt(37))):
        a = np.array(v)
        assert bound.pair_ratio(a.ctypes.data_as(ctypes.c_void_p), len(a)) == pytest.approx(want)


def _runs(bound, s, eps_max):
    run, runs = 0, [0]
    for a, b in zip(s[:-1], s[1:]):
        run += not bound.tie(a, b, eps_max)
        runs.append(run)
    return runs


def test_open_ranks_are_closed_under_their_bounds(bound):
    """Scores of different runs are certain against each other, whatever the bounds in between: a wide bound beside
    narrow ones on either side, then random lists."""
    cases = [([1.00, 0.99, 0.95], [0.10, 0.001, 0.001]), ([1.00, 0.97, 0.96], [0.001, 0.001, 0.10])]
    rng = np.random.default_rng(5)
    for _ in range(200):
        n = int(rng.integers(2, 40))
        cases.append((np.sort(rng.uniform(0, 1, n))[::-1], 10.0 ** rng.uniform(-5, -1.5, n)))
    for s, e in cases:
        runs = _runs(bound, list(map(float, s)), float(max(e)))
        for a in range(len(s)):
            for b in range(a + 1, len(s)):
                assert runs[a] == runs[b] or s[a] - s[b] > e[a] + e[b]
    assert len(set(_runs(bound, [1.00, 0.99, 0.95], 0.10))) == 1  # (0.99 and 0.95 are certain, 1.00 and 0.95 are not)
