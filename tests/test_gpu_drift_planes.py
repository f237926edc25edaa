"""Drift correction at the window sizes where the plane kernels' passes, batches and
padding change (padded sides 2 to 256, flat z, one window and many), against the oracle's
restatement in double precision.  Tolerance as tests/test_gpu_drift.py: the library's
transforms are single precision, so a pair's peak centroid moves by a small fraction of a
voxel."""
import numpy as np
import pytest

import oracle as O
from test_oracle import drift_data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,bins,L,Lz", [
    (4, 3, 300.0, 100.0), (8, 4, 700.0, 200.0), (16, 3, 400.0, 300.0),  # many small windows: batches
    (16, 3, 400.0, 0.0), (32, 3, 500.0, 150.0), (64, 2, 700.0, 60.0),   # flat z; unequal sides
    (128, 2, 1500.0, 30.0),                                             # planes of 256 x 256: axis by axis
    (16, 2, 90.0, 60.0)])                                               # a single window, cut to the data
def test_drift_windows_match_oracle(zpkg, ctx, size, bins, L, Lz):
    xyz, fr, cr, dt, vel = drift_data(seed=size + bins, nf=500, nbead=30, n_per=40, L=L, Lz=max(Lz, 1.0),
                                      vel=(0.02, -0.01, 0.005 if Lz else 0.0))
    if Lz == 0:
        xyz[:, 2] = 0.0
    kw = dict(pixel_nm=10.0, bins=bins, max_drift_um=size * 0.01)
    got_b, got_l, px = zpkg.drift(ctx, xyz, fr, cr, **kw)
    want_b, want_l, wpx = O.drift(xyz, fr, cr, **kw)
    again_b, again_l, _ = zpkg.drift(ctx, xyz, fr, cr, **kw)
    assert px == wpx
    assert np.array_equal(got_b, again_b) and np.array_equal(got_l, again_l)
    assert np.array_equal(got_b[:, 0], want_b[:, 0])
    assert np.abs(got_b[:, 1:] - want_b[:, 1:]).max() < 0.05 * px
    assert np.abs(got_l - want_l).max() < 0.1 * px
