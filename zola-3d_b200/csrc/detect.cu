// PSF-library cross-correlation detection (process/cpu/Predetection.java:63-593).
//
// Per frame (S_x x S_y photons, first index x):
//   k_det_rowsum, k_det_colsum, k_det_var
//                local mean / variance over the R-wide box by the reference's
//                running sums (Predetection.java:337-405), operation for
//                operation (no FMA contraction), on the float-rounded image
//   scores       normalised cross-correlation with the zero-mean library PSFs.
//                The reference multiplies unitary FFTs on a zero-padded M x M
//                grid (M = pow2(2S)); with that padding the product is the
//                linear correlation corr(i,j) = sum_uv img[i+u-R/2][j+v-R/2]
//                psf0[u][v], scaled by 1/sqrt(Mx My): score = corr / sqrt(varPSF
//                * varImage) (-1 / -2 where a variance is not positive,
//                :459-471).  FP64 FFTs (detect_fft.cu) screen the candidates;
//                small windows, and frames on which the FFT's rounding could
//                change a decision, take the direct sum (k_det_corr_rt,
//                k_det_corr).  Returned scores are direct sums either way.
//   k_det_peaks  per slice r: tmp = max over j +- 3 where score > 0 (tmp keeps
//                the previous slice's value elsewhere, as the reference reuses
//                it), then peaks with score > thr equal to tmp and to the max of
//                tmp over i +- 3 (:480-560)
//   k_det_emit   the candidates in the reference's insertion order (r, then j,
//                then i), so the stored list is the same on every run
//   k_det_refine rows score, r, i, j, topZ, topX, topY with parabolic x/y/z
//                refinement, from direct sums
//   k_det_sort   stable sort by descending score (Arrays.sort of the rows in
//                insertion order r, j, i; :447-454): ties keep list order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "det_bound.h"
#include "zola_internal.h"

namespace zola {



// ---------------------------------------------------------------------------
// Running sums exactly as Predetection.setImage: first along y for every x,
// then along x for every y.  Double arithmetic with explicit rounding
// intrinsics so the compiler cannot fuse multiply-adds.  A running sum is a
// serial chain, so the three kernels keep everything else off it: the chain's
// operands arrive in shared memory or registers a block of 32 (8) steps ahead,
// and the divisions are a pass of their own.  One CTA a frame with strided reads
// and the divisions in the chain took 128 us for one 130^2 frame and 421 us for
// 48 frames of 256^2.

// s1, s2: running sums of the float-rounded image and of its square along y, a
// CTA for 32 rows.  Warp 0 runs the chains (lane = row) over 32 columns while the
// other warps fetch the next 32 and write out the last.  amax[f]: the bits of
// the largest |pixel| (above those of infinity where a pixel is not a number).
constexpr int VR_ROWS = 32, VR_THREADS = 128, VR_S = VR_ROWS + 1;
constexpr int VR_SMEM = 4 * VR_ROWS * VR_S * 4 + 4 * VR_ROWS * VR_S * 8;

__global__ void __launch_bounds__(VR_THREADS) k_det_rowsum(DetView V, const double* frames, double* rowsum,
                                                           double* rowsq, unsigned long long* amax) {
    extern __shared__ __align__(16) char vsm[];
    double* outs = (double*)vsm;                       // [buffer][sum, square][row][column]
    float* ins = (float*)(outs + 4 * VR_ROWS * VR_S);  // [buffer][leaving, entering][row][column]
    const int f = blockIdx.y, SX = V.SX, SY = V.SY, h = V.R / 2, i0 = blockIdx.x * VR_ROWS;
    const int nr = min(VR_ROWS, SX - i0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* img = frames + (size_t)f * SX * SY + (size_t)i0 * SY;
    double* s1 = rowsum + (size_t)f * SX * SY + (size_t)i0 * SY;
    double* s2 = rowsq + (size_t)f * SX * SY + (size_t)i0 * SY;
    unsigned long long m = 0;
    for (int k = threadIdx.x; k < nr * SY; k += VR_THREADS)
        m = max(m, (unsigned long long)__double_as_longlong(fabs(img[k])));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) atomicMax(&amax[f], m);
    // Line t < 2 nr: row t % nr of the leaving (t < nr) or entering pixels.  A warp takes
    // every nt-th line, eight loads in flight.
    constexpr int U = 8;
    auto fetch = [&](int c, int t0, int nt) {
        for (int tb = t0; tb < 2 * nr; tb += U * nt) {
            float x[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int t = tb + q * nt, e = t >= nr, col = 32 * c + lane + (e ? h : -h);
                x[q] = t < 2 * nr && col >= 0 && col < SY ? (float)img[(size_t)(t - e * nr) * SY + col] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const int t = tb + q * nt, e = t >= nr;
                if (t < 2 * nr) ins[(((c & 1) * 2 + e) * VR_ROWS + t - e * nr) * VR_S + lane] = x[q];
            }
        }
    };
    const int nc = (SY + 31) / 32;
    fetch(0, warp, VR_THREADS / 32);
    double a = 0.0, b = 0.0;
    if (warp == 0 && lane < nr)
        for (int t = 0; t < h + 1; ++t)
            if (t < SY) {
                const double x = (double)(float)img[(size_t)lane * SY + t];
                a = __dadd_rn(a, x);
                b = __dadd_rn(b, __dmul_rn(x, x));
            }
    __syncthreads();
    for (int c = 0; c <= nc; ++c) {
        if (warp == 0) {
            if (c < nc && lane < nr) {
                const float* lv = ins + ((c & 1) * 2 * VR_ROWS + lane) * VR_S;
                const float* en = lv + VR_ROWS * VR_S;
                double* oa = outs + ((c & 1) * 2 * VR_ROWS + lane) * VR_S;
                double* ob = oa + VR_ROWS * VR_S;
#pragma unroll 8
                for (int t = 0; t < 32; ++t) {
                    const int ii = 32 * c + t;
                    if (ii > 0) {
                        if (ii - h >= 0) { const double x = lv[t]; a = __dsub_rn(a, x); b = __dsub_rn(b, __dmul_rn(x, x)); }
                        if (ii + h < SY) { const double x = en[t]; a = __dadd_rn(a, x); b = __dadd_rn(b, __dmul_rn(x, x)); }
                    }
                    oa[t] = a;
                    ob[t] = b;
                }
            }
        } else {
            if (c + 1 < nc) fetch(c + 1, warp - 1, VR_THREADS / 32 - 1);
            if (c > 0)
                for (int t = warp - 1; t < 2 * nr; t += VR_THREADS / 32 - 1) {
                    const int e = t >= nr, row = t - e * nr, col = 32 * (c - 1) + lane;
                    if (col < SY)
                        (e ? s2 : s1)[(size_t)row * SY + col] =
                            outs[((((c - 1) & 1) * 2 + e) * VR_ROWS + row) * VR_S + lane];
                }
        }
        __syncthreads();
    }
}

// The running sums of s1 and s2 along x, a thread a column; the operands of the
// next 8 rows are loaded before the chain of these 8 runs.
__global__ void __launch_bounds__(32) k_det_colsum(DetView V, const double* rowsum, const double* rowsq, double* sum,
                                                   double* sq) {
    const int SX = V.SX, SY = V.SY, h = V.R / 2, ii = blockIdx.x * 32 + threadIdx.x;
    if (ii >= SY) return;
    const size_t base = (size_t)blockIdx.y * SX * SY + ii;
    const double *s1 = rowsum + base, *s2 = rowsq + base;
    constexpr int U = 8;
    double n1[U], n2[U], p1[U], p2[U];  // entering, leaving
    auto load = [&](int i0) {
#pragma unroll
        for (int t = 0; t < U; ++t) {
            const int e = i0 + t + h, l = i0 + t - h;
            n1[t] = e < SX ? s1[(size_t)e * SY] : 0.0;
            n2[t] = e < SX ? s2[(size_t)e * SY] : 0.0;
            p1[t] = l >= 0 && l < SX ? s1[(size_t)l * SY] : 0.0;
            p2[t] = l >= 0 && l < SX ? s2[(size_t)l * SY] : 0.0;
        }
    };
    double a = 0.0, b = 0.0;
    for (int t = 0; t < h + 1; ++t)
        if (t < SX) { a = __dadd_rn(a, s1[(size_t)t * SY]); b = __dadd_rn(b, s2[(size_t)t * SY]); }
    load(0);
    for (int i0 = 0; i0 < SX; i0 += U) {
        double c1[U], c2[U], d1[U], d2[U];
#pragma unroll
        for (int t = 0; t < U; ++t) { c1[t] = n1[t]; c2[t] = n2[t]; d1[t] = p1[t]; d2[t] = p2[t]; }
        if (i0 + U < SX) load(i0 + U);
#pragma unroll
        for (int t = 0; t < U; ++t) {
            const int i = i0 + t;
            if (i >= SX) break;
            if (i > 0) {
                if (i - h >= 0) { a = __dsub_rn(a, d1[t]); b = __dsub_rn(b, d2[t]); }
                if (i + h < SX) { a = __dadd_rn(a, c1[t]); b = __dadd_rn(b, c2[t]); }
            }
            sum[base + (size_t)i * SY] = a;
            sq[base + (size_t)i * SY] = b;
        }
    }
}

// Bound of |FFT score - directly summed score| at a pixel: k max|pixel| /
// sqrt(varImage) + base (det_fft_bound).
struct DetEps {
    double k, base;
    const unsigned long long* amax;  // bits of max|pixel| per frame (k_det_rowsum)
    const double* isv;               // 1 / sqrt(varImage), -1 where the variance is not positive
};

// In place: sum -> variance of the box, sq -> isv.  With marks, inexact[f] is set
// where a pixel of frame f is not finite or the bound of a score that a candidate is
// compared with exceeds DET_EPS_MAX (camera frames have 1e-8 and less), the slack of
// k_det_look.
constexpr double DET_EPS_MAX = 1e-4;
__global__ void __launch_bounds__(256) k_det_var(DetView V, double* sum, double* sq, DetEps E, int* inexact) {
    const size_t SS = (size_t)V.SX * V.SY;
    const int f = blockIdx.y, lo = max(3, V.R / 2);
    const double kf = inexact ? E.k * __longlong_as_double((long long)E.amax[f]) : 0.0;
    bool bad = !(kf < INFINITY);
    for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < SS; k += (size_t)gridDim.x * 256) {
        const double n = V.norm[k], mean = __ddiv_rn(sum[f * SS + k], n);
        const double v = __dsub_rn(__ddiv_rn(sq[f * SS + k], n), __dmul_rn(mean, mean)), w = v > 0 ? 1.0 / sqrt(v) : -1.0;
        sum[f * SS + k] = v;
        sq[f * SS + k] = w;
        const int i = (int)(k / V.SY), j = (int)(k - (size_t)i * V.SY);
        // (k_det_look compares candidates with the three columns on either side of the inner part)
        if (i >= lo && i < V.SX - lo && j >= lo - 3 && j < V.SY - lo + 3) bad |= !(kf * w + E.base < DET_EPS_MAX);
    }
    if (inexact && bad) inexact[f] = 1;
}

// The score of a correlation sum.
__device__ inline double det_score(const DetView& V, double corr, double vp, double vi) {
    const double s = sqrt(vp * vi);
    if (s > 0) return (corr * V.inv_m) / s;
    return vp <= 0 ? -1.0 : -2.0;
}

// ---------------------------------------------------------------------------
// Direct FP64 correlation of a 16 x 16 output tile against ZC slices.
constexpr int DT = 16;
constexpr int ZC = 8;

// only (nullable): the frames with only[f] != 0.
__global__ void __launch_bounds__(256) k_det_corr(DetView V, int zc, const double* frames, const double* var,
                                                  double* score, const int* only) {
    extern __shared__ double sm[];
    const int SX = V.SX, SY = V.SY, R = V.R, Z = V.Z, h = R / 2, TW = DT + R;
    const int f = blockIdx.z;
    if (only && !only[f]) return;
    const int z0 = blockIdx.y * zc;
    const int tiles_y = (SY + DT - 1) / DT;
    const int i0 = (blockIdx.x / tiles_y) * DT, j0 = (blockIdx.x % tiles_y) * DT;
    double* tile = sm;               // TW x TW image with halo
    double* ps = tile + TW * TW;     // ZC x R x R
    const double* img = frames + (size_t)f * SX * SY;
    for (int k = threadIdx.x; k < TW * TW; k += blockDim.x) {
        const int a = k / TW, b = k % TW;
        const int i = i0 - h + a, j = j0 - h + b;
        tile[k] = (i >= 0 && i < SX && j >= 0 && j < SY) ? img[(size_t)i * SY + j] : 0.0;
    }
    const int nz = min(zc, Z - z0);
    for (int k = threadIdx.x; k < nz * R * R; k += blockDim.x) ps[k] = V.psf0[(size_t)z0 * R * R + k];
    __syncthreads();
    const int ti = threadIdx.x / DT, tj = threadIdx.x % DT;
    const int i = i0 + ti, j = j0 + tj;
    double acc[ZC];
#pragma unroll
    for (int q = 0; q < ZC; ++q) acc[q] = 0.0;
    for (int u = 0; u < R; ++u) {
        const double* trow = tile + (ti + u) * TW + tj;
        for (int v = 0; v < R; ++v) {
            const double x = trow[v];
#pragma unroll
            for (int q = 0; q < ZC; ++q)
                if (q < nz) acc[q] = fma(x, ps[(q * R + u) * R + v], acc[q]);
        }
    }
    if (i >= SX || j >= SY) return;
    const double vi = var[(size_t)f * SX * SY + (size_t)i * SY + j];
    for (int q = 0; q < nz; ++q) {
        const int r = z0 + q;
        score[(((size_t)f * Z + r) * SX + i) * SY + j] = det_score(V, acc[q], V.varpsf[r], vi);
    }
}

// ---------------------------------------------------------------------------
// Register-tiled form of the same correlation (same terms, same order per
// output: u outer, v inner, one FMA each), bound by the FP64 FMA pipe instead
// of shared-memory loads.  A CTA of 256 threads covers a 32 x 64 output tile
// and RZC slices; each thread owns 8 consecutive outputs of one row for every
// slice (32 accumulators).  For each kernel row u a thread keeps an 8-wide
// window of the image row in registers and slides it along v, so one image
// load and RZC broadcast library loads feed 8 RZC FMAs.  A half-warp holds
// 16 consecutive rows of one 8-column group; with an odd row stride their
// window loads fall in 16 different bank pairs.
constexpr int RTI = 32, RTJ = 64, RPX = 8, RZC = 4;

__host__ __device__ inline int rt_stride(int R) { return (RTJ + R) | 1; }
__host__ __device__ inline size_t rt_smem(int R, int zc) {
    return (size_t)(RTI + R) * rt_stride(R) * 8 + (size_t)zc * R * R * 8;
}

__global__ void __launch_bounds__(256, 2) k_det_corr_rt(DetView V, int zc, const double* frames, const double* var,
                                                         double* score, const int* only) {
    extern __shared__ double sm[];
    const int SX = V.SX, SY = V.SY, R = V.R, Z = V.Z, h = R / 2, TS = rt_stride(R), TH = RTI + R;
    const int f = blockIdx.z, z0 = blockIdx.y * zc;
    if (only && !only[f]) return;
    const int tiles_j = (SY + RTJ - 1) / RTJ;
    const int i0 = (blockIdx.x / tiles_j) * RTI, j0 = (blockIdx.x % tiles_j) * RTJ;
    double* tile = sm;                    // (RTI + R) rows x TS (RTJ + R used, zero-filled)
    double* ps = tile + (size_t)TH * TS;  // zc x R x R
    const double* img = frames + (size_t)f * SX * SY;
    const int TW = RTJ + R;  // the last window load (v = R - 1) reads column RTJ + R - 1
    for (int k = threadIdx.x; k < TH * TW; k += blockDim.x) {
        const int a = k / TW, b = k - a * TW;
        const int i = i0 - h + a, j = j0 - h + b;
        tile[a * TS + b] = (i >= 0 && i < SX && j >= 0 && j < SY) ? img[(size_t)i * SY + j] : 0.0;
    }
    const int nz = min(zc, Z - z0);
    for (int k = threadIdx.x; k < nz * R * R; k += blockDim.x) ps[k] = V.psf0[(size_t)z0 * R * R + k];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ti = (lane & 15) + 16 * (warp & 1), tj = 8 * (2 * (warp >> 1) + (lane >> 4));
    double acc[RZC][RPX];
#pragma unroll
    for (int q = 0; q < RZC; ++q)
#pragma unroll
        for (int k = 0; k < RPX; ++k) acc[q][k] = 0.0;
    const int RR = R * R;
    for (int u = 0; u < R; ++u) {
        const double* trow = tile + (ti + u) * TS + tj;
        const double* prow = ps + u * R;
        double w[RPX];
#pragma unroll
        for (int k = 0; k < RPX; ++k) w[k] = trow[k];
        // unrolled by the window width: the window's shifts become register renames
#pragma unroll 8
        for (int v = 0; v < R; ++v) {
            double p[RZC];
#pragma unroll
            for (int q = 0; q < RZC; ++q) p[q] = q < nz ? prow[q * RR + v] : 0.0;
#pragma unroll
            for (int q = 0; q < RZC; ++q)
#pragma unroll
                for (int k = 0; k < RPX; ++k) acc[q][k] = fma(w[k], p[q], acc[q][k]);
#pragma unroll
            for (int k = 0; k < RPX - 1; ++k) w[k] = w[k + 1];
            w[RPX - 1] = trow[v + RPX];
        }
    }
    const int i = i0 + ti;
    if (i >= SX) return;
    for (int k = 0; k < RPX; ++k) {
        const int j = j0 + tj + k;
        if (j >= SY) break;
        const double vi = var[(size_t)f * SX * SY + (size_t)i * SY + j];
#pragma unroll
        for (int q = 0; q < RZC; ++q) {
            if (q >= nz) break;
            const int r = z0 + q;
            score[(((size_t)f * Z + r) * SX + i) * SY + j] = det_score(V, acc[q][k], V.varpsf[r], vi);
        }
    }
}

// ---------------------------------------------------------------------------
// Camera counts to photons as LocalizationPipeline.java:601-605 does it:
// value * (adu / gain) + (-offset * adu / gain), a product then a sum (Java
// does not contract them), negative results set to 0.
__global__ void k_u16_photons(const uint16_t* in, size_t n, double slope, double intercept, double* out) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const double v = __dadd_rn(__dmul_rn((double)in[k], slope), intercept);
        out[k] = v < 0 ? 0.0 : v;
    }
}

void rescale_u16(zola_ctx* ctx, const uint16_t* d_in, size_t n, const double* rescale, double* d_out,
                 cudaStream_t st) {
    k_u16_photons<<<ctx->num_sms * 8, 256, 0, st>>>(d_in, n, rescale[0], rescale[1], d_out);
    ctx->launches++;
}

void camera_rescale(double adu, double gain, double offset, double* rescale) {
    rescale[0] = adu / gain;            // rescale_slope (LocalizationPipeline.java:103)
    rescale[1] = -offset * adu / gain;  // rescale_intercept (:104)
}

// ---------------------------------------------------------------------------
__device__ inline double parabola_top(double xa, double ya, double xb, double yb, double xc, double yc) {
    const double a = (yc - ya) / ((xc - xa) * (xc - xb)) - (yb - ya) / ((xb - xa) * (xc - xb));
    const double b = ((yb - ya) / (xb - xa)) - a * (xb + xa);
    return -b / (2 * a);
}

// Exclusive prefix sum of one int per thread over the block, in thread order;
// *total = the block's sum.  wtot: 32 ints of shared memory.
__device__ int block_exclusive_scan(int v, int* wtot, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wtot[w] = x;
    __syncthreads();
    if (w == 0) {
        int y = lane < nw ? wtot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += u;
        }
        if (lane < nw) wtot[lane] = y;
    }
    __syncthreads();
    const int base = w ? wtot[w - 1] : 0;
    *total = wtot[nw - 1];
    __syncthreads();  // wtot is reused by the next call
    return base + x - v;
}

// ---------------------------------------------------------------------------
// Peaks.  The reference keeps tmp, the maximum over j +- 3, per pixel and only
// overwrites it where the slice's score is positive; a pixel is a peak when its
// score is above thr, equals its own tmp, and no tmp of i +- 3 is larger.  So
// the tmp that slice r sees at a pixel is the one of the last slice r' <= r with
// a positive score there (0: none, or outside the border), which any thread can
// find by itself: slices need no order, and only pixels that pass the first two
// tests look at their column.
//
// Two kernels: k_det_look reads every score once and leaves one pixel in some
// 200, which k_det_peaks tests in full.  48 frames of 256^2 x 40 take 340 + 515 us,
// of which reading the scores alone is 160; in one kernel, 1.2 ms, the full tests'
// registers halved the warps of the first look, and a third of the lanes ran most
// of the instructions.  (One CTA a frame, slice after slice: 6.4 ms.)
//
// Scores of the FFT correlation are within eps (DetEps) of the direct sum's.  A
// decision that eps could turn marks the frame in inexact[]; marked frames are taken again with directly summed
// scores (again = 1, eps = 0).  inexact = nullptr: every score is the direct sum's.
// bits: a bit per (slice, j, i), 32 values of i to a word; tot: peaks per slice.

// First look, a warp a row: sets the bits of the pixels above the threshold that no
// score within three pixels of the row or the column exceeds, with room for both
// bounds and for the row's single precision.  56 pixels at a time, two a lane: one
// in 20 passes the row's test, and 32 of those at a time read their column.
__global__ void __launch_bounds__(256) k_det_look(DetView V, const double* score, const int* inexact, int again,
                                                  unsigned* bits) {
    const int f = blockIdx.z, r = blockIdx.y, SX = V.SX, SY = V.SY, dec = 3, lo = max(dec, V.R / 2);
    const int i = lo + blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const bool approx = inexact && !again;
    if (inexact && again && !inexact[f]) return;
    if (i >= SX - lo) return;
    const double* row = score + (((size_t)f * V.Z + r) * SX + i) * SY;
    const int WX = (SX + 31) / 32, jend = SY - lo;
    unsigned* out = bits + ((size_t)f * V.Z + r) * SY * WX + (i >> 5);
    constexpr double SLACK = 3e-4;  // more than two eps (DET_EPS_MAX) and the rounding
    __shared__ short keep[8][96];
    short* mine = keep[threadIdx.x >> 5];
    int n = 0;
    auto column = [&]() {  // the first min(n, 32) pixels of the list
        const int j = mine[lane];
        double c[2 * dec + 1];
#pragma unroll
        for (int k = 0; k <= 2 * dec; ++k) c[k] = lane < n ? row[(ptrdiff_t)(k - dec) * SY + j] : 0.0;
        bool stay = lane < n;
#pragma unroll
        for (int k = 0; k <= 2 * dec; ++k) {
            const int ic = i + k - dec;
            if (k != dec && ic >= lo && ic < SX - lo && c[k] > 0 && c[k] > c[dec] + SLACK) stay = false;
        }
        if (stay) atomicOr(out + (size_t)j * WX, 1u << (i & 31));
        const int rest = max(n - 32, 0);
        short t[2];
        for (int k = 0; k < 2; ++k) t[k] = mine[min(32 + 32 * k + lane, 95)];
        __syncwarp();
        for (int k = 0; k < 2; ++k) mine[32 * k + lane] = t[k];
        n = rest;
        __syncwarp();
    };
    const float thr = approx ? (float)(V.thr - SLACK) : __double2float_rd(V.thr);
    auto load = [&](int j) { return j >= lo - dec && j < jend + dec ? (float)row[j] : -INFINITY; };
    float an = load(lo - 4 + 2 * lane), bn = load(lo - 3 + 2 * lane);
    for (int j0 = lo; j0 < jend; j0 += 56) {
        const int j = j0 - 4 + 2 * lane;
        const float a = an, b = bn, m = fmaxf(a, b);
        an = load(j + 56);
        bn = load(j + 57);
        const unsigned all = 0xffffffffu;
        const float ml = __shfl_up_sync(all, m, 1), mr = __shfl_down_sync(all, m, 1);
        const float bl = __shfl_up_sync(all, b, 2), ar = __shfl_down_sync(all, a, 2);
        const float side = fmaxf(ml, mr), na = fmaxf(side, fmaxf(bl, b)), nb = fmaxf(side, fmaxf(ar, a));
        const bool mid = lane >= 2 && lane < 30;
        auto passes = [&](float v, float w, int jj) {
            const bool beaten = w > v + (float)SLACK + 1e-6f * fabsf(v) && (approx || v > 0);
            return mid && jj < jend && (approx ? v > thr : v >= thr) && !beaten;
        };
        const bool pa = passes(a, na, j), pb = passes(b, nb, j + 1);
        const unsigned ba = __ballot_sync(all, pa), bb = __ballot_sync(all, pb), below = (1u << lane) - 1;
        if (pa) mine[n + __popc(ba & below)] = (short)j;
        n += __popc(ba);
        if (pb) mine[n + __popc(bb & below)] = (short)(j + 1);
        n += __popc(bb);
        __syncwarp();
        while (n >= 32) column();
    }
    if (n > 0) column();
}

// The full tests of the pixels that k_det_look left, a word of bits a lane.
__global__ void __launch_bounds__(256) k_det_peaks(DetView V, const double* score, DetEps E, int* inexact, int again,
                                                   unsigned* bits, int* tot) {
    const int f = blockIdx.z, r = blockIdx.y, SX = V.SX, SY = V.SY, Z = V.Z, dec = 3, lo = max(dec, V.R / 2);
    const int WX = (SX + 31) / 32, word = blockIdx.x * 256 + threadIdx.x, lane = threadIdx.x & 31;
    const size_t SS = (size_t)SX * SY;
    const bool approx = inexact && !again;
    if (inexact && again && !inexact[f]) return;
    unsigned* at_word = bits + ((size_t)f * Z + r) * SY * WX + word;
    const unsigned seen = word < SY * WX ? *at_word : 0;
    if (!__any_sync(0xffffffffu, seen != 0)) return;
    const double kf = approx ? E.k * __longlong_as_double((long long)E.amax[f]) : 0.0;
    const double* sc = score + (size_t)f * Z * SS;
    const double* iv = approx ? E.isv + f * SS : nullptr;
    auto eps_at = [&](int ic, int jc) { return approx ? kf * fmax(iv[(size_t)ic * SY + jc], 0.0) + E.base : 0.0; };
    // The tests of pixel (i, j) against its row and the column's scores, a lane a pixel.
    auto test = [&](int i, int j, double& v, double& eps, bool& unsure) {
        const double* row = sc + (size_t)r * SS + (size_t)i * SY;
        v = row[j];
        eps = eps_at(i, j);
        if (!(v + eps > V.thr)) return false;
        unsure = !(v - eps > V.thr);
        bool peak = true;
        auto beats = [&](double w, double ew) {  // w against the candidate
            if (w - ew > v + eps) peak = false;
            else if (approx && w + ew >= v - eps) unsure = true;
        };
        // the row's and the column's scores first (a positive score is below its own tmp)
        double cs[2 * dec], ce[2 * dec];
#pragma unroll
        for (int k = 0; k < 2 * dec; ++k) {
            const int a = k < dec ? -1 - k : k - dec + 1;
            cs[k] = row[(ptrdiff_t)a * SY + j];
            ce[k] = eps_at(i + a, j);
            if (approx || v > 0) beats(row[j + a], eps_at(i, j + a));
        }
#pragma unroll
        for (int k = 0; k < 2 * dec; ++k) {
            const int ic = i + (k < dec ? -1 - k : k - dec + 1);
            if (ic >= lo && ic < SX - lo && cs[k] > ce[k] && cs[k] - ce[k] > v + eps) peak = false;
        }
        if (!peak) return false;
        if (!approx && !(v > 0)) {  // its own tmp is an earlier slice's, or 0
            double t = 0.0;
            for (int q = r - 1; q >= 0; --q) {
                const double* s = sc + (size_t)q * SS + (size_t)i * SY + j;
                if (!(*s > 0)) continue;
                t = -INFINITY;
                for (int a = -dec; a <= dec; ++a) t = fmax(s[a], t);
                break;
            }
            if (v != t) return false;
        }
        return true;
    };
    // Candidate (i, j) against the tmp of (ic, j) as slice r sees it, for the six ic: zero,
    // or seven scores' maximum.  By the whole warp: a lane a slice, since the last slice
    // with a positive score can be far below r, then a lane a score.  0: not a peak, 1: a
    // peak, 2: a peak if the scores were exact.
    auto against_tmp = [&](int i, int j, double v, double eps, bool unsure) {
        bool beaten = false;
        auto beats = [&](double w, double ew) {
            if (w - ew > v + eps) beaten = true;
            else if (approx && w + ew >= v - eps) unsure = true;
        };
        int at[2 * dec];  // that slice, or -1
        double e[2 * dec];
        unsigned open = 0;
#pragma unroll
        for (int k = 0; k < 2 * dec; ++k) {
            const int ic = i + (k < dec ? -1 - k : k - dec + 1);
            at[k] = -1;
            e[k] = 0.0;
            if (ic >= lo && ic < SX - lo) {
                open |= 1u << k;
                e[k] = eps_at(ic, j);
            }
        }
        for (int q0 = r; q0 >= 0 && open; q0 -= 32) {
            double x[2 * dec];
#pragma unroll
            for (int k = 0; k < 2 * dec; ++k) {
                const int ic = i + (k < dec ? -1 - k : k - dec + 1);
                x[k] = (open >> k & 1) && q0 - lane >= 0 ? sc[(size_t)(q0 - lane) * SS + (size_t)ic * SY + j] : -INFINITY;
            }
#pragma unroll
            for (int k = 0; k < 2 * dec; ++k) {
                const unsigned pos = __ballot_sync(0xffffffffu, x[k] > e[k]);
                if (approx && (open >> k & 1) && x[k] > -e[k] && (pos & ((2u << lane) - 1)) == 0) unsure = true;
                if (pos) {
                    at[k] = q0 - (__ffs(pos) - 1);
                    open &= ~(1u << k);
                }
            }
        }
        int z = -1, d = 0;
        for (int p = lane; p < 2 * dec * (2 * dec + 1); p += 32) {
            const int k = p / (2 * dec + 1), c = k < dec ? -1 - k : k - dec + 1;
#pragma unroll
            for (int m = 0; m < 2 * dec; ++m)
                if (m == k) z = at[m];
            d = p - k * (2 * dec + 1) - dec;
            if (z >= 0) beats(sc[(size_t)z * SS + (size_t)(i + c) * SY + j + d], eps_at(i + c, j + d));
            else beats(0.0, 0.0);
        }
        if (__any_sync(0xffffffffu, beaten)) return 0;
        return approx && __any_sync(0xffffffffu, unsure) ? 2 : 1;
    };
    unsigned left = seen, peaks = 0;
    while (__any_sync(0xffffffffu, left != 0)) {
        const int bit = left ? __ffs(left) - 1 : 0, i = word % WX * 32 + bit, j = word / WX;
        double v = 0, eps = 0;
        bool unsure = false;
        unsigned alive = __ballot_sync(0xffffffffu, left && test(i, j, v, eps, unsure));
        left &= left - 1;
        for (; alive; alive &= alive - 1) {
            const int k = __ffs(alive) - 1;
            const int is = against_tmp(__shfl_sync(0xffffffffu, i, k), __shfl_sync(0xffffffffu, j, k),
                                       __shfl_sync(0xffffffffu, v, k), __shfl_sync(0xffffffffu, eps, k),
                                       __shfl_sync(0xffffffffu, unsure, k));
            if (is == 1 && lane == k) peaks |= 1u << bit;
            if (is == 2 && lane == 0) inexact[f] = 1;
        }
    }
    if (peaks != seen) *at_word = peaks;
    const int found = __reduce_add_sync(0xffffffffu, __popc(peaks));
    if (lane == 0 && found) atomicAdd(&tot[(size_t)f * Z + r], found);
}

// Clears the peaks of the marked frames before their second pass.
__global__ void __launch_bounds__(256) k_det_unmark(DetView V, const int* inexact, unsigned* bits, int* tot) {
    const int f = blockIdx.y;
    if (!inexact[f]) return;
    const size_t n = (size_t)V.Z * V.SY * ((V.SX + 31) / 32);
    for (size_t k = (size_t)blockIdx.x * 256 + threadIdx.x; k < n; k += (size_t)gridDim.x * 256) bits[f * n + k] = 0;
    for (int k = blockIdx.x * 256 + threadIdx.x; k < V.Z; k += gridDim.x * 256) tot[(size_t)f * V.Z + k] = 0;
}

// Candidates of one slice of one frame (a CTA): score as the volume holds it,
// slice, i, j, in the reference's insertion order: slice, column j, row i.  The
// first V.cap rows of the frame's list are stored; counts[f] = the length of the
// whole list.
__global__ void __launch_bounds__(128) k_det_emit(DetView V, const double* score, const unsigned* bits, const int* tot,
                                                  double* cand, int* counts) {
    __shared__ int wtot[32];
    const int r = blockIdx.x, f = blockIdx.y, SX = V.SX, SY = V.SY, Z = V.Z, lo = max(3, V.R / 2);
    const int WX = (SX + 31) / 32;
    int before = 0, base;
    for (int q = threadIdx.x; q < r; q += blockDim.x) before += tot[(size_t)f * Z + q];
    block_exclusive_scan(before, wtot, &base);
    const int n = tot[(size_t)f * Z + r];
    if (r == Z - 1 && threadIdx.x == 0) counts[f] = base + n;
    const double* sc = score + ((size_t)f * Z + r) * SX * SY;
    double* out = cand + (size_t)f * V.cap * 7;
    for (int j0 = lo; n > 0 && j0 < SY - lo; j0 += blockDim.x) {
        const int j = j0 + threadIdx.x;
        const unsigned* w = bits + (((size_t)f * Z + r) * SY + min(j, SY - 1)) * WX;
        int c = 0, all;
        if (j < SY - lo)
            for (int q = 0; q < WX; ++q) c += __popc(w[q]);
        int o = base + block_exclusive_scan(c, wtot, &all);
        if (c)
            for (int q = 0; q < WX; ++q)
                for (unsigned b = w[q]; b; b &= b - 1, ++o)
                    if (o < V.cap) {
                        const int i = 32 * q + __ffs(b) - 1;
                        double* t = out + (size_t)o * 7;
                        t[0] = sc[(size_t)i * SY + j]; t[1] = r; t[2] = i; t[3] = j;
                    }
        base += all;
    }
}

// ---------------------------------------------------------------------------
// Score and parabolic offsets of candidates, from the correlations at the pixel
// and its six neighbours (r -+ 1, i -+ 1, j -+ 1), each summed directly in the order
// of k_det_corr (u outer, v inner, one FMA each): the rows are the direct form's
// bit for bit, whatever screened them.
// A warp takes four candidates, eight lanes each; lanes 0-6 own one of the seven
// sums.  A sum is a serial chain of R^2 FMAs, so everything else is kept off it:
// image rows (a ring) and library rows (double buffered) come into shared memory by
// cp.async, the next four rows while these four are summed.  With the library rows
// read through L1 instead, 768 candidates at R = 40 took 120 us, bound by their
// latency.
constexpr int DR_WARPS = 2, DR_BLOCK = 4, DR_RING = 2 * DR_BLOCK + 2;
__host__ __device__ inline int refine_stride(int R) { return R + 3; }  // odd
__host__ __device__ inline int refine_doubles(int R) {  // per candidate
    return 2 * DR_BLOCK * 3 * R + DR_RING * refine_stride(R);
}
__host__ __device__ inline size_t refine_smem(int R) { return (size_t)DR_WARPS * 4 * refine_doubles(R) * sizeof(double); }

// The candidate row t of frame f, for this lane's group of eight (every lane of
// the warp takes part; a group without a candidate passes another one's row and
// store = false).
__device__ void refine_row(const DetView& V, const double* frames, const double* var, int f, double* t, bool store) {
    extern __shared__ __align__(16) char esm[];
    const int SX = V.SX, SY = V.SY, R = V.R, h = R / 2, lane = threadIdx.x & 31, q = lane & 7;
    const size_t SS = (size_t)SX * SY;
    const double* img = frames + f * SS;
    const int r = (int)t[1], i = (int)t[2], j = (int)t[3];
    const bool zin = r > 1 && r < V.Z - 1;
    // this lane's sum: slice r + dr at pixel (i + di, j + dj) (lane 7 repeats lane 0)
    const int dr = zin ? (q == 2) - (q == 1) : 0, di = (q == 4) - (q == 3), dj = (q == 6) - (q == 5);
    const int P = refine_stride(R);
    double* lib = (double*)esm + (size_t)(threadIdx.x >> 3) * refine_doubles(R);  // [buffer][row][slice][column]
    double* ring = lib + 2 * DR_BLOCK * 3 * R;
    const unsigned lib_s = (unsigned)__cvta_generic_to_shared(lib), ring_s = (unsigned)__cvta_generic_to_shared(ring);
    const double* src = img + (ptrdiff_t)(i - 1 - h) * SY + (j - 1 - h);
    const double* p0 = V.psf0 + (size_t)max(r - 1, 0) * R * R;
    const double* p1 = V.psf0 + (size_t)r * R * R;
    const double* p2 = V.psf0 + (size_t)min(r + 1, V.Z - 1) * R * R;
    // image rows i - 1 - h + a for a0 <= a < a1, columns j - 1 - h .. j + h, zeros outside the frame
    auto fetch_image = [&](int a0, int a1) {
        for (int a = a0; a < min(a1, R + 2); ++a) {
            const int ic = i - 1 - h + a;
            const unsigned dst = ring_s + (a % DR_RING) * P * 8;
            for (int v = q; v < R + 2; v += 8) {
                const bool in = ic >= 0 && ic < SX && j - 1 - h + v >= 0 && j - 1 - h + v < SY;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst + v * 8),
                             "l"(in ? src + (ptrdiff_t)a * SY + v : img), "r"(in ? 8 : 0)
                             : "memory");
            }
        }
    };
    // library rows u0 .. u0 + 3 of the three slices (R is even: rows are whole 16-byte pieces)
    auto fetch_library = [&](int u0) {
        for (int u = u0; u < min(u0 + DR_BLOCK, R); ++u) {
            const unsigned dst = lib_s + ((u / DR_BLOCK & 1) * DR_BLOCK + u % DR_BLOCK) * 3 * R * 8;
            for (int v = q; v < R / 2; v += 8) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + v * 16), "l"(p0 + u * R + 2 * v)
                             : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (R * 8) + v * 16),
                             "l"(p1 + u * R + 2 * v)
                             : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (2 * R * 8) + v * 16),
                             "l"(p2 + u * R + 2 * v)
                             : "memory");
            }
        }
    };
    double acc = 0.0;
    fetch_image(0, DR_BLOCK + 2);
    fetch_library(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int u0 = 0; u0 < R; u0 += DR_BLOCK) {
        fetch_image(u0 + DR_BLOCK + 2, u0 + 2 * DR_BLOCK + 2);
        fetch_library(u0 + DR_BLOCK);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        for (int u = u0; u < min(u0 + DR_BLOCK, R); ++u) {
            const double* x = ring + ((u + 1 + di) % DR_RING) * P + 1 + dj;
            const double* p = lib + (((u / DR_BLOCK & 1) * DR_BLOCK + u % DR_BLOCK) * 3 + 1 + dr) * R;
            int v = 0;
            for (; v + 8 <= R; v += 8) {
                double xs[8], ws[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) { xs[k] = x[v + k]; ws[k] = p[v + k]; }
#pragma unroll
                for (int k = 0; k < 8; ++k) acc = fma(xs[k], ws[k], acc);
            }
            for (; v < R; ++v) acc = fma(x[v], p[v], acc);
        }
        __syncwarp();  // the rows of this block are overwritten next
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    const double s = det_score(V, acc, V.varpsf[r + dr], var[f * SS + (size_t)(i + di) * SY + j + dj]);
    const int l0 = lane & 24;
    const double s0 = __shfl_sync(0xffffffffu, s, l0), sl = __shfl_sync(0xffffffffu, s, l0 + min(2 * q + 1, 5)),
                 sh = __shfl_sync(0xffffffffu, s, l0 + min(2 * q + 2, 6));
    if (store && q < 4) {  // lanes 0-2: the offset along z, x, y; lane 3: the score
        if (q == 3) t[0] = s0;
        else if (q == 0) t[4] = zin ? parabola_top(-V.zstep, sl, 0, s0, V.zstep, sh) : 0.0;
        else t[4 + q] = parabola_top(-V.dx, sl, 0, s0, V.dx, sh);
    }
}

// The candidates of rank 0 .. want - 1 of every frame (order: list positions by
// rank), or, with order = nullptr, of list positions 0 .. want - 1.
__global__ void __launch_bounds__(32 * DR_WARPS) k_det_refine(DetView V, const double* frames, const double* var,
                                                              double* cand, const int* counts, const int* order, int want) {
    const int f = blockIdx.y, n = min(min(counts[f], V.cap), want);
    for (int g = blockIdx.x * DR_WARPS * 4; g < n; g += gridDim.x * DR_WARPS * 4) {
        const int w = g + (threadIdx.x >> 5) * 4, k = w + ((threadIdx.x & 31) >> 3);
        if (w >= n) continue;  // the whole warp
        const int e = min(k, n - 1), p = order ? order[(size_t)f * V.cap + e] : e;
        refine_row(V, frames, var, f, cand + ((size_t)f * V.cap + p) * 7, k < n);
    }
}

// The same for n candidates (n_dev: read there) of any frames, cand[frame][index].
__global__ void __launch_bounds__(32 * DR_WARPS) k_det_refine_list(DetView V, const double* frames, const double* var,
                                                                   double* cand, int n, const int* n_dev,
                                                                   const int* frame, const int* index) {
    if (n_dev) n = *n_dev;
    for (int g = blockIdx.x * DR_WARPS * 4; g < n; g += gridDim.x * DR_WARPS * 4) {
        const int w = g + (threadIdx.x >> 5) * 4, k = w + ((threadIdx.x & 31) >> 3);
        if (w >= n) continue;
        const int e = min(k, n - 1);
        refine_row(V, frames, var, frame[e], cand + ((size_t)frame[e] * V.cap + index[e]) * 7, k < n);
    }
}

// Sort keys of up to DET_SORT_SMEM candidates per frame live in shared memory;
// longer lists sort in global scratch (same network).
constexpr int DET_SORT_SMEM = 16384;

__host__ __device__ inline int det_pow2(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Sort one frame's stored candidates by (score descending, list position
// ascending) -- a stable sort of the insertion-ordered list: order[f][rank] =
// list position.  gs / gid: global sort keys (det_pow2(cap) per frame) or nullptr
// for the shared-memory form.
// D.count (nullable): where screening scores next to each other in the order are
// too close for it to be certain (det_tie), both candidates are listed (D.frame, D.index)
// and the pair is marked (D.tie[f][rank]: rank and rank + 1).  k_det_ties orders them.
struct DetTies {
    int *count, *frame, *index;
    unsigned char* tie;
};
__global__ void __launch_bounds__(1024) k_det_sort(DetView V, const double* cand, const int* counts, int* order, double* gs,
                                                   int* gid, DetEps E, const int* inexact, DetTies D) {
    extern __shared__ double smraw[];
    __shared__ unsigned long long eps_bits;
    const int f = blockIdx.x, n = min(counts[f], V.cap);
    const int P2 = det_pow2(n);
    double* s = gs ? gs + (size_t)f * det_pow2(V.cap) : smraw;
    int* id = gs ? gid + (size_t)f * det_pow2(V.cap) : (int*)(smraw + P2);
    const double* c = cand + (size_t)f * V.cap * 7;
    for (int t = threadIdx.x; t < P2; t += blockDim.x) {
        if (t < n) { s[t] = c[(size_t)t * 7]; id[t] = t; }
        else { s[t] = -INFINITY; id[t] = 0x7fffffff; }
    }
    if (threadIdx.x == 0) eps_bits = 0;
    __syncthreads();
    // the largest bound of the list (positive: its bits are in its order)
    const bool screened = D.count && !inexact[f];
    if (screened) {
        const double kf = E.k * __longlong_as_double((long long)E.amax[f]);
        double m = 0.0;
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const double* r = c + (size_t)t * 7;
            m = fmax(m, kf * fmax(E.isv[((size_t)f * V.SX + (int)r[2]) * V.SY + (int)r[3]], 0.0) + E.base);
        }
        atomicMax(&eps_bits, (unsigned long long)__double_as_longlong(m));
    }
    // bitonic network: "before" = higher score, then earlier in the list
    for (int size = 2; size <= P2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < P2; t += blockDim.x) {
                const int o = t ^ stride;
                if (o > t) {
                    const bool up = (t & size) == 0;
                    const bool t_before = s[t] > s[o] || (s[t] == s[o] && id[t] < id[o]);
                    if (up != t_before) {
                        const double ts = s[t]; s[t] = s[o]; s[o] = ts;
                        const int ti = id[t]; id[t] = id[o]; id[o] = ti;
                    }
                }
            }
            __syncthreads();
        }
    __syncthreads();
    const double eps_max = __longlong_as_double((long long)eps_bits);
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        order[(size_t)f * V.cap + t] = id[t];
        if (!D.count) continue;
        const bool tie = screened && t + 1 < n && det_tie(s[t], s[t + 1], eps_max);
        D.tie[(size_t)f * V.cap + t] = tie;
        if (tie) {  // (the middle of a longer run is listed twice, with the same result)
            const int o = atomicAdd(D.count, 2);
            D.frame[o] = D.frame[o + 1] = f;
            D.index[o] = id[t];
            D.index[o + 1] = id[t + 1];
        }
    }
}

// Orders each run of marked ranks by the direct scores (ties by list position): a
// thread a run, nearly always a pair.  Scores outside a run are certain against it
// (det_tie).
__global__ void __launch_bounds__(256) k_det_ties(DetView V, const double* cand, const int* counts, int* order,
                                                  const unsigned char* tie) {
    const int f = blockIdx.y, n = min(counts[f], V.cap);
    const unsigned char* m = tie + (size_t)f * V.cap;
    int* o = order + (size_t)f * V.cap;
    const double* c = cand + (size_t)f * V.cap * 7;
    for (int t = blockIdx.x * 256 + threadIdx.x; t < n; t += gridDim.x * 256) {
        if (!m[t] || (t > 0 && m[t - 1])) continue;
        for (int e = t + 1; e < n && m[e - 1]; ++e) {
            const int p = o[e];
            const double s = c[(size_t)p * 7];
            int k = e;
            for (; k > t; --k) {
                const int p2 = o[k - 1];
                const double s2 = c[(size_t)p2 * 7];
                if (s2 > s || (s2 == s && p2 < p)) break;
                o[k] = p2;
            }
            o[k] = p;
        }
    }
}

// Rows by rank: the first `rows` of each frame's list to out[f][rank].
__global__ void __launch_bounds__(256) k_det_gather(DetView V, const double* cand, const int* counts, const int* order,
                                                    int rows, double* out) {
    const int f = blockIdx.y, n = min(min(counts[f], V.cap), rows);
    for (int t = blockIdx.x * 256 + threadIdx.x; t < n * 7; t += gridDim.x * 256) {
        const int row = t / 7, col = t - row * 7;
        out[(size_t)f * V.cap * 7 + t] = cand[((size_t)f * V.cap + order[(size_t)f * V.cap + row]) * 7 + col];
    }
}

// Which detectors screen by FFT.  Thresholds near or below zero (where most of
// the frame is a candidate, and the sign of a score decides) and small windows
// keep the direct sum, whose cost falls with R^2.  Whole detect calls, direct
// against FFT, us: 32 frames of 128^2 x 40 slices 1773 / 1638 at R = 12, 1986 /
// 1584 at R = 16, 2442 / 1402 at R = 24; one frame of 64^2 x 8 slices 154 / 162,
// 156 / 161, 196 / 165; 48 frames of 256^2 x 40 at R = 40 18.6 ms / 4.8 ms.
bool det_fft_wanted(const DetView& v) { return v.thr >= 1e-3 && v.R >= DET_FFT_MIN_R; }

}  // namespace zola

// ------------------------------------------------------------------ host ----

using namespace zola;

extern "C" {

int zola_detector_create(zola_psf* psf, int SX, int SY, int R, double minZ, double maxZ, double step, double thr,
                         zola_detector** out) {
    if (!psf || !out) return ZOLA_E_ARG;
    zola_ctx* ctx = psf->ctx;
    *out = nullptr;
    if (SX < 8 || SY < 8 || SX > 4096 || SY > 4096 || R < 4 || R % 2 || R > SX || R > SY || R > 96 || !(step > 0) ||
        !(maxZ > minZ)) {
        ctx->err = "zola_detector_create: need 8 <= S <= 4096, even R <= min(S, 96), step > 0, maxZ > minZ";
        return ZOLA_E_ARG;
    }
    int number = (int)std::ceil((maxZ - minZ) / step);  // Predetection.java:120-127
    if (number < 1 || number > 4096) { ctx->err = "zola_detector_create: bad number of library slices"; return ZOLA_E_ARG; }
    zola_detector* d = new zola_detector();
    d->psf = psf;
    double z = minZ;
    for (int i = 0; i < number; ++i) { d->range.push_back(z); z += step; }
    // library PSFs with the FP64 model: x = y = 0, zoil = Zfocus, zwat = range[i]
    d->h_psf.resize((size_t)number * R * R);
    int rc = library_psfs(psf, R, d->range.data(), number, d->h_psf.data());
    if (rc) { delete d; return rc; }
    std::vector<double> psf0((size_t)number * R * R), varpsf(number), norm((size_t)SX * SY);
    for (int i = 0; i < number; ++i) {  // Predetection.java:178-204
        const double* p = d->h_psf.data() + (size_t)i * R * R;
        double mean = 0;
        for (int k = 0; k < R * R; ++k) mean += p[k];
        mean /= (double)R * R;
        double v = 0;
        for (int k = 0; k < R * R; ++k) {
            double q = p[k] - mean;
            psf0[(size_t)i * R * R + k] = q;
            v += q * q;
        }
        varpsf[i] = v / (double)(R * R);
    }
    for (int i = 0; i < SX; ++i)  // Predetection.java:95-116 (index rules kept)
        for (int ii = 0; ii < SY; ++ii) {
            int vx1 = R / 2, vx2 = R / 2, vy1 = R / 2, vy2 = R / 2;
            if (i < R / 2 - 1) vx1 = i + 1;
            if (i > SX - R / 2 - 2) vx2 = SY - i - 1;
            if (ii < R / 2 - 1) vy1 = ii + 1;
            if (ii > SX - R / 2 - 2) vy2 = SY - ii - 2;
            norm[(size_t)i * SY + ii] = (double)((vx1 + vx2) * (vy1 + vy2));
        }
    size_t total = psf0.size() + varpsf.size() + norm.size();
    cudaError_t e = cudaMalloc(&d->d_lib, total * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpy(d->d_lib, psf0.data(), psf0.size() * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d->d_lib + psf0.size(), varpsf.data(), varpsf.size() * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(d->d_lib + psf0.size() + varpsf.size(), norm.data(), norm.size() * 8, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        ctx->err = std::string("zola_detector_create: ") + cudaGetErrorString(e);
        if (d->d_lib) cudaFree(d->d_lib);
        delete d;
        return ZOLA_E_CUDA;
    }
    int MX = 1, MY = 1;
    while (MX < 2 * SX) MX <<= 1;
    while (MY < 2 * SY) MY <<= 1;
    DetView& v = d->v;
    v.SX = SX; v.SY = SY; v.R = R; v.Z = number; v.cap = 0;
    v.inv_m = 1.0 / std::sqrt((double)MX * (double)MY);
    v.thr = thr; v.zstep = step; v.dx = psf->o.xystep;
    v.psf0 = d->d_lib; v.varpsf = d->d_lib + psf0.size(); v.norm = d->d_lib + psf0.size() + varpsf.size();
    det_fft_build(ctx, v, d->fft);
    d->fft.pair = det_pair_ratio(varpsf.data(), number);
    *out = d;
    return ZOLA_OK;
}

int zola_detector_free(zola_detector* d) {
    if (!d) return ZOLA_E_ARG;
    cudaStreamSynchronize(d->psf->ctx->stream);
    cudaFree(d->d_lib);
    det_fft_free(d->fft);
    delete d;
    return ZOLA_OK;
}

int zola_detector_info(const zola_detector* d, int* nslices, double* range, double* psfs) {
    if (!d || !nslices) return ZOLA_E_ARG;
    *nslices = d->v.Z;
    if (range)
        for (int i = 0; i < d->v.Z; ++i) range[i] = d->range[i];
    if (psfs)
        for (size_t k = 0; k < d->h_psf.size(); ++k) psfs[k] = d->h_psf[k];
    return ZOLA_OK;
}

int zola_detect_dev(zola_detector* d, const double* d_frames, int nframes, int cap, double* d_out, int* d_counts,
                    void* stream) {
    if (!d) return ZOLA_E_ARG;
    zola_ctx* ctx = d->psf->ctx;
    if (nframes < 0 || cap < 1 || cap > ZOLA_DETECT_MAX_CAP || (nframes > 0 && (!d_frames || !d_out || !d_counts))) {
        ctx->err = "zola_detect: bad nframes / cap (1..2^20) or null buffer";
        return ZOLA_E_ARG;
    }
    return detect_frames(d, d_frames, nframes, cap, cap, cap, d_out, d_counts, nullptr,
                         stream ? (cudaStream_t)stream : ctx->stream);
}

}  // extern "C"

namespace zola {

// Candidate lists of device frames: `cap` rows are stored per frame; the first
// `rows` of them go to d_out[f][cap][7] by rank, the first `want` of these with
// directly summed scores and offsets (the others have the screening's score and no
// offsets; detect_refine completes rows by index).  d_var (nullable): the frames'
// box variances, for detect_refine.
int detect_frames(zola_detector* d, const double* d_frames, int nframes, int cap, int rows, int want, double* d_out,
                  int* d_counts, double* d_var, cudaStream_t st) {
    zola_ctx* ctx = d->psf->ctx;
    if (nframes == 0) return ZOLA_OK;
    DetView v = d->v;
    v.cap = cap;
    const size_t SS = (size_t)v.SX * v.SY;
    const int p2 = det_pow2(cap);
    const bool gsort = p2 > DET_SORT_SMEM;
    bool fft = d->fft.d_tab != nullptr;
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    // scratch per frame: row sums and their squares, variance, its inverse root, scores
    // (Z x SS), candidates, peak bits and counts, and the sort keys when they do not fit
    // in shared memory; for the FFT correlation also the spectra
    const size_t bits_b = (size_t)v.Z * v.SY * ((v.SX + 31) / 32) * 4;
    int chunk = 0;
    for (;; fft = false) {
        const size_t per = (4 + (size_t)v.Z) * SS * 8 + (size_t)cap * (7 * 8 + 4 + 17) + bits_b + (size_t)v.Z * 4 + 12 +
                           (gsort ? (size_t)p2 * 12 : 0) +
                           (fft ? (size_t)d->fft.MY * (v.SX + d->fft.MX) * sizeof(double2) : 0);
        chunk = (int)std::max<size_t>(1, std::min<size_t>(std::min(nframes, 65535), ((size_t)1 << 31) / per));
        if (ensure_scratch(ctx, per * chunk + (fft ? det_fft_scratch(v, d->fft, 1) + DET_FFT_T_BYTES : 0) + 8192, ctx->err) == 0)
            break;
        if (!fft) return ZOLA_E_CUDA;
        cudaGetLastError();  // no room for the spectra: direct sums, which give the same rows
    }
    const size_t rsmem = refine_smem(v.R), ssort = gsort ? 0 : (size_t)p2 * 12;
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_det_rowsum, cudaFuncAttributeMaxDynamicSharedMemorySize, VR_SMEM), ctx);
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_det_refine, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem), ctx);
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_det_refine_list, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem), ctx);
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_det_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssort), ctx);
    for (int f0 = 0; f0 < nframes; f0 += chunk) {
        const int nf = std::min(chunk, nframes - f0);
        char* b = (char*)ctx->scratch;
        auto take = [&](size_t bytes) { char* q = b; b += al(bytes); return q; };
        double* rowsum = (double*)take(nf * SS * 8);
        double* rowsq = (double*)take(nf * SS * 8);
        double* var = d_var ? d_var + f0 * SS : (double*)take(nf * SS * 8);
        double* isv = (double*)take(nf * SS * 8);
        double* score = (double*)take(nf * v.Z * SS * 8);
        double* cand = (double*)take((size_t)nf * cap * 7 * 8);
        // cleared together: peak bits, peaks per slice, largest |pixel|, marks
        char* zero = b;
        unsigned* bits = (unsigned*)take(nf * bits_b);
        int* tot = (int*)take((size_t)nf * v.Z * 4);
        unsigned long long* amax = (unsigned long long*)take((size_t)nf * 8);
        int* inexact = (int*)take((size_t)nf * 4);
        DetTies D{(int*)take(4), nullptr, nullptr, nullptr};
        const size_t zero_b = b - zero;
        int* order = (int*)take((size_t)nf * cap * 4);
        D.frame = (int*)take((size_t)nf * cap * 8);
        D.index = (int*)take((size_t)nf * cap * 8);
        D.tie = (unsigned char*)take((size_t)nf * cap);
        double* gs = gsort ? (double*)take((size_t)nf * p2 * 8) : nullptr;
        int* gid = gsort ? (int*)take((size_t)nf * p2 * 4) : nullptr;
        const double* fr = d_frames + (size_t)f0 * SS;
        ZOLA_CUDA_CHECK(cudaMemsetAsync(zero, 0, zero_b, st), ctx);
        prof_begin(ctx, 9, st);
        k_det_rowsum<<<dim3((v.SX + VR_ROWS - 1) / VR_ROWS, nf), VR_THREADS, VR_SMEM, st>>>(v, fr, rowsum, rowsq, amax);
        k_det_colsum<<<dim3((v.SY + 31) / 32, nf), 32, 0, st>>>(v, rowsum, rowsq, var, isv);
        DetEps E{0, 0, amax, isv};
        if (fft) det_fft_bound(v.SX, v.SY, v.R, d->fft.MX, d->fft.MY, v.inv_m, d->fft.pair, &E.k, &E.base);
        k_det_var<<<dim3((unsigned)std::min<size_t>((SS + 255) / 256, 256), nf), 256, 0, st>>>(v, var, isv, E,
                                                                                              fft ? inexact : nullptr);
        ctx->launches += 3;
        auto direct = [&](const int* only) {
            // slices per register-tiled CTA: as many (up to RZC) as keep two CTAs per SM
            int zrt = RZC;
            while (zrt > 0 && rt_smem(v.R, zrt) > 112 * 1024) --zrt;
            if (zrt > 0) {
                const int tiles = ((v.SX + RTI - 1) / RTI) * ((v.SY + RTJ - 1) / RTJ);
                const size_t smem = rt_smem(v.R, zrt);
                cudaFuncSetAttribute(k_det_corr_rt, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                dim3 grid(tiles, (v.Z + zrt - 1) / zrt, nf);
                k_det_corr_rt<<<grid, 256, smem, st>>>(v, zrt, fr, var, score, only);
            } else {
                const int tiles = ((v.SX + DT - 1) / DT) * ((v.SY + DT - 1) / DT);
                const size_t tile_b = (size_t)(DT + v.R) * (DT + v.R) * 8, slice_b = (size_t)v.R * v.R * 8;
                const int zc = (int)std::max<size_t>(1, std::min<size_t>(ZC, (200 * 1024 - tile_b) / slice_b));
                const size_t smem = tile_b + (size_t)zc * slice_b;
                cudaFuncSetAttribute(k_det_corr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                dim3 grid(tiles, (v.Z + zc - 1) / zc, nf);
                k_det_corr<<<grid, 256, smem, st>>>(v, zc, fr, var, score, only);
            }
            ctx->launches++;
        };
        const int lo = std::max(3, v.R / 2);
        auto peaks = [&](int* marks, int again) {
            const unsigned rows = (unsigned)std::max(1, (v.SX - 2 * lo + 7) / 8);
            k_det_look<<<dim3(rows, v.Z, nf), 256, 0, st>>>(v, score, marks, again, bits);
            const unsigned words = (unsigned)v.SY * ((v.SX + 31) / 32);
            k_det_peaks<<<dim3((words + 255) / 256, v.Z, nf), 256, 0, st>>>(v, score, E, marks, again, bits, tot);
            ctx->launches += 2;
        };
        if (fft) {
            det_fft_scores(ctx, v, d->fft, fr, nf, isv, b, score, st);
            peaks(inexact, 0);
            direct(inexact);  // the frames that the screening could not decide
            k_det_unmark<<<dim3(32, nf), 256, 0, st>>>(v, inexact, bits, tot);
            peaks(inexact, 1);
            ctx->launches++;
        } else {
            direct(nullptr);
            peaks(nullptr, 0);
        }
        int* cnt = d_counts + f0;
        k_det_emit<<<dim3(v.Z, nf), 128, 0, st>>>(v, score, bits, tot, cand, cnt);
        const int per_cta = 4 * DR_WARPS;
        auto refine = [&](const int* by_rank, int first) {
            const unsigned gx = (unsigned)std::max(1, std::min((first + per_cta - 1) / per_cta, 64 * ctx->num_sms / nf + 1));
            k_det_refine<<<dim3(gx, nf), 32 * DR_WARPS, rsmem, st>>>(v, fr, var, cand, cnt, by_rank, first);
        };
        if (!fft || want >= cap) {  // every row: refined in list order, where neighbours share their slice
            refine(nullptr, cap);
            D.count = nullptr;
            k_det_sort<<<nf, 1024, ssort, st>>>(v, cand, cnt, order, gs, gid, E, inexact, D);
        } else {  // rank by the screening's scores, directly where those leave a doubt
            k_det_sort<<<nf, 1024, ssort, st>>>(v, cand, cnt, order, gs, gid, E, inexact, D);
            k_det_refine_list<<<ctx->num_sms, 32 * DR_WARPS, rsmem, st>>>(v, fr, var, cand, 0, D.count, D.frame, D.index);
            k_det_ties<<<dim3(8, nf), 256, 0, st>>>(v, cand, cnt, order, D.tie);
            if (want > 0) refine(order, want);
            ctx->launches += 2;
        }
        k_det_gather<<<dim3((unsigned)std::min((rows * 7 + 255) / 256, 64), nf), 256, 0, st>>>(
            v, cand, cnt, order, rows, d_out + (size_t)f0 * cap * 7);
        prof_end(ctx, st);
        ctx->launches += 3;
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { ctx->err = std::string("zola_detect: ") + cudaGetErrorString(e); return ZOLA_E_CUDA; }
    }
    return ZOLA_OK;
}

int detect_refine(zola_detector* d, const double* d_frames, const double* d_var, double* d_cand, int cap, int n,
                  const int* d_frame, const int* d_index, cudaStream_t st) {
    zola_ctx* ctx = d->psf->ctx;
    if (n <= 0) return ZOLA_OK;
    DetView v = d->v;
    v.cap = cap;
    const size_t smem = refine_smem(v.R);
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_det_refine_list, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), ctx);
    k_det_refine_list<<<(n + 4 * DR_WARPS - 1) / (4 * DR_WARPS), 32 * DR_WARPS, smem, st>>>(v, d_frames, d_var, d_cand, n,
                                                                                           nullptr, d_frame, d_index);
    ctx->launches++;
    ZOLA_CUDA_CHECK(cudaGetLastError(), ctx);
    return ZOLA_OK;
}

}  // namespace zola

namespace {

// frames (photons) or u16 camera counts with rescale = {slope, intercept}
int detect_impl(zola_detector* d, const double* frames, const uint16_t* u16, const double* rescale, int nframes,
                int cap, double* out, int* counts) {
    if (!d) return ZOLA_E_ARG;
    zola_ctx* ctx = d->psf->ctx;
    if (nframes < 0 || cap < 1 || cap > ZOLA_DETECT_MAX_CAP ||
        (nframes > 0 && ((!frames && !u16) || !out || !counts))) {
        ctx->err = "zola_detect: bad nframes / cap (1..2^20) or null buffer";
        return ZOLA_E_ARG;
    }
    if (nframes == 0) return ZOLA_OK;
    const size_t SS = (size_t)d->v.SX * d->v.SY;
    // Candidates stored per frame in the first pass: at least DETECT_ROOM, so that the
    // usual lists (a few thousand at the reference's threshold) are whole and sorted
    // in one pass whatever cap the caller asks for.
    constexpr int DETECT_ROOM = 8192;
    const int room0 = std::max(cap, DETECT_ROOM);
    // frames, counts, the uint16 frames and the candidate rows come from the
    // context's grow-only staging area, so repeated calls allocate nothing
    auto al = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t b_df = al(SS * nframes * 8), b_dc = al((size_t)nframes * 4), b_du = u16 ? al(SS * nframes * 2) : 0;
    if (ensure_io(ctx, b_df + b_dc + b_du + al((size_t)nframes * room0 * 7 * 8))) return ZOLA_E_CUDA;
    char* io = (char*)ctx->io;
    double* df = (double*)io;
    int* dc = (int*)(io + b_df);
    uint16_t* du = u16 ? (uint16_t*)(io + b_df + b_dc) : nullptr;
    double* dout = (double*)(io + b_df + b_dc + b_du);
    cudaError_t e = cudaSuccess;
    if (u16) {
        e = copy_in(ctx, du, u16, SS * nframes * 2, ctx->stream);
        if (e == cudaSuccess) rescale_u16(ctx, du, SS * nframes, rescale, df, ctx->stream);
    } else {
        e = copy_in(ctx, df, frames, SS * nframes * 8, ctx->stream);
    }
    int rc = e == cudaSuccess ? detect_frames(d, df, nframes, room0, cap, cap, dout, dc, nullptr, ctx->stream) : ZOLA_OK;
    if (e == cudaSuccess && rc == ZOLA_OK) {
        e = cudaMemcpyAsync(counts, dc, (size_t)nframes * 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    // A frame whose list is longer than the room kept the first candidates in scan
    // order, not the best: such frames are gathered and detected again with room
    // for their whole lists, and the first cap rows of each replace theirs.
    std::vector<int> longf;
    int room = room0;
    if (e == cudaSuccess && rc == ZOLA_OK)
        for (int f = 0; f < nframes; ++f)
            if (counts[f] > room0) {
                longf.push_back(f);
                room = std::max(room, counts[f]);
            }
    double* g = nullptr;  // gathered frames, their rows, their counts (rare: one allocation)
    if (!longf.empty() && room > ZOLA_DETECT_MAX_CAP) {
        ctx->err = "zola_detect: a frame has more than 2^20 candidates";
        rc = ZOLA_E_ARG;
    } else if (!longf.empty()) {
        const size_t nl = longf.size();
        e = cudaMalloc(&g, nl * SS * 8 + nl * (size_t)room * 7 * 8 + nl * 4);
        double* g_out = g + nl * SS;
        int* g_cnt = (int*)(g_out + nl * (size_t)room * 7);
        for (size_t k = 0; k < nl && e == cudaSuccess; ++k)
            e = cudaMemcpyAsync(g + k * SS, df + (size_t)longf[k] * SS, SS * 8, cudaMemcpyDeviceToDevice, ctx->stream);
        if (e == cudaSuccess) rc = detect_frames(d, g, (int)nl, room, cap, cap, g_out, g_cnt, nullptr, ctx->stream);
        for (size_t k = 0; k < nl && e == cudaSuccess && rc == ZOLA_OK; ++k)
            e = cudaMemcpyAsync(dout + (size_t)longf[k] * room0 * 7, g_out + k * room * 7, (size_t)cap * 7 * 8,
                                cudaMemcpyDeviceToDevice, ctx->stream);
    }
    if (e == cudaSuccess && rc == ZOLA_OK) {
        e = cudaMemcpy2DAsync(out, (size_t)cap * 7 * 8, dout, (size_t)room0 * 7 * 8, (size_t)cap * 7 * 8, nframes,
                              cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    if (g) {
        cudaStreamSynchronize(ctx->stream);
        cudaFree(g);
    }
    if (e != cudaSuccess) { ctx->err = std::string("zola_detect: ") + cudaGetErrorString(e); return ZOLA_E_CUDA; }
    return rc;
}

}  // namespace

extern "C" {

int zola_detect(zola_detector* d, const double* frames, int nframes, int cap, double* out, int* counts) {
    return detect_impl(d, frames, nullptr, nullptr, nframes, cap, out, counts);
}

int zola_detect_u16(zola_detector* d, const uint16_t* frames, int nframes, int cap, double adu, double gain,
                    double offset, double* out, int* counts) {
    if (!d) return ZOLA_E_ARG;
    if (!(gain != 0) || !std::isfinite(adu) || !std::isfinite(gain) || !std::isfinite(offset)) {
        d->psf->ctx->err = "zola_detect_u16: adu, gain, offset must be finite and gain non-zero";
        return ZOLA_E_ARG;
    }
    double rescale[2];
    camera_rescale(adu, gain, offset, rescale);
    return detect_impl(d, nullptr, frames, rescale, nframes, cap, out, counts);
}

}  // extern "C"
