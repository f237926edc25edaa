"""The operation counts that the bench divides by its times are those of the forms that run."""
import math

import numpy as np

import bench


def test_detection_counts_line_transforms():
    line = 5 * 288 * math.log2(288)  # 256 + 20 padded to 288 points
    both = 256 * line + 288 * line
    want = both + 21 * (both + 6 * 288 * 288) + 3 * 41 * 256 * 256
    assert math.isclose(bench.detect_flops(256, 256, 40, 41), want, rel_tol=1e-12)
    assert want < 0.1 * 2 * 256 * 256 * 40 * 40 * 41  # (a direct sum for every pixel)


def test_fp64_fits_count_the_trial_and_what_is_summed_again():
    fft, direct = bench.fft_eval_flops(24, 128), bench.direct_eval_flops(24, 128)
    assert fft < 0.25 * direct
    status, evals = np.array([1, 1, 2]), np.array([7, 20, 50])
    assert math.isclose(bench.fp64_fit_flops(24, 128, status, evals), fft * (7 + 12 + 12) + direct * 70, rel_tol=1e-12)
