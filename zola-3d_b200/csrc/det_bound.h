// What the FFT correlation of the detection may decide by itself: the bound of its
// scores' error, and the ranks that it leaves open.  Plain arithmetic, host and device.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define DET_FN __host__ __device__ inline
#else
#define DET_FN inline
#endif

namespace zola {

// The largest ratio of the norm of two slices that share a complex transform (2 p and
// 2 p + 1) to that of one of them.  var: the slices' variances; where one is not positive
// its scores are fixed, and the other has the transform to itself.
DET_FN double det_pair_ratio(const double* var, int Z) {
    double most = 1.0;
    for (int r = 0; r + 1 < Z; r += 2)
        if (var[r] > 0 && var[r + 1] > 0) {
            const double less = var[r] < var[r + 1] ? var[r] : var[r + 1], ratio = std::sqrt((var[r] + var[r + 1]) / less);
            if (!(ratio <= most)) most = ratio;
        }
    return most;
}

// Bound of |FFT score - directly summed score| = k max|pixel| / sqrt(varImage) + base, of
// SX x SY frames with R x R slices on an MX x MY grid; inv_m: the scores' scale; pair:
// det_pair_ratio.  Three transforms with relative 2-norm errors of at most
// 5 u log2(MX MY) each (u = 2^-53), ||img|| <= sqrt(SX SY) max|pixel|, for the pair
// ||psf0|| = pair R sqrt(varPSF), and |FFT(psf0)| <= R ||psf0|| (the inverse transform's
// part); the direct sum's own rounding, at most R^2 u sum |img psf0|; and a few roundings
// of the score's scaling, |score| <= R^2 / sqrt(Mx My).
DET_FN void det_fft_bound(int SX, int SY, int R_, int MX, int MY, double inv_m, double pair, double* k, double* base) {
    const double u = std::ldexp(1.0, -53), R = R_;
    const double fft = 15 * u * std::log2((double)MX * MY) * (1 + R) * std::sqrt((double)SX * SY) * R * pair;
    *k = (fft + u * R * R * R * R) * inv_m;
    *base = 32 * u * (1 + R * R * inv_m);
}

// Whether two scores next to each other in the order of the screening belong to one run
// of open ranks.  eps_max: the largest bound in the list, so that scores of different runs
// are more than any two bounds apart, whichever of a run's they are.
DET_FN bool det_tie(double s, double next, double eps_max) { return s - next <= 2 * eps_max; }

}  // namespace zola
