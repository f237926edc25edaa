// Frame localization pipeline: detection -> candidate selection -> fit ->
// filters and mask -> localization rows (process/cpu/LocalizationPipeline.java).
//
// The reference walks each frame's sorted candidate list on a Java thread
// (LocalizationThread.run, LocalizationPipeline.java:720-990):
//   - next candidate whose centre pixel is unmasked and inside the border
//     (myGetMaxPositions, :1218-1250);
//   - skip it if any pixel of its R x R patch is masked;
//   - getAandB init from the library PSF of its slice (:1119-1162); fit only
//     if maxPatch / B > maxSNR (1) and B > 0, else mask the patch pixels above
//     half the patch maximum;
//   - accept if A > photonThreshold, |x|,|y| < 10 px, the rounded position is
//     inside the frame and unmasked, and minZ < z < maxZ (:859-945); then mask
//     the pixels where model - B > 0.2 max(model - B);
//   - otherwise mask the patch pixels above half the patch maximum (:967-977).
// A candidate's fit reads only the raw patch and its getAandB start, never
// the mask, so the fits do not depend on the order.  Frames advance in waves:
// each wave takes, per frame, the next K candidates that need a fit under the
// current mask (one CTA per frame tests candidates in parallel chunks: border,
// centre and patch masks, getAandB, SNR), completes their starts, fits all of them in one batched call
// (FP64 or split), evaluates the model at every fitted position, and then one
// CTA per frame replays the reference's sequential walk over the candidates
// the wave covered: mask tests, acceptance, mask updates.  A candidate masked
// by an earlier one in the same wave was fitted for nothing; masks only grow,
// so a candidate the wave found masked stays skipped.  Accepted localizations
// get chi2 as scoreCompute (:1099-1115) and the CRLB from the Fisher matrix the
// reference forms (Localization.java:317-451: dmu/dA taken as mu, h -> 0
// limit).  Rows come out in frame order and, within a frame, in candidate
// order; x/y/z in nm as 1000*(i*dx - x) (:905-907).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "lm.h"
#include "zola_internal.h"

namespace zola {

struct PipeView {
    int SX, SY, R, cap, nframes;
    double dx, minZ, maxZ, photon_thr, max_snr;
    const double* images;     // nframes x SX x SY: detection images
    const double* fimg;       // nframes x SX x SY: fit images (= images without sCMOS)
    const double* vmap;       // SX x SY sCMOS var/gain^2, or nullptr
    float* slot_v;            // slots x R x R sCMOS patches (with vmap)
    unsigned char* mask;      // nframes x SX x SY
    unsigned* near_mask;      // nframes x SX x ceil(SY / 32): a bit per pixel whose R x R patch has a masked pixel
    const double* cand;       // nframes x cap x 7
    const int* counts;        // nframes
    const double* libpsf;     // Z x R x R (normalised library PSFs)
    const double* range;      // Z
    int* cand_slot;           // nframes x cap: fit slot; -1 not fitted (SNR), -2 outside the border,
                              // -3 masked when the wave looked at it
    double* cand_maxp;        // nframes x cap: patch maximum
    int* pointer;             // nframes: first candidate not yet walked
    int* limit;               // nframes: end of the candidates the current wave covers
    int* done;                // nframes
    int* nslots;              // slots of the current wave
    int slot_cap;
    float* rois;              // slots x R x R
    double* init;             // slots x 5
    int* slot_frame;          // slots
    int* slot_cand;           // slots
};

__device__ inline bool pipe_inside(const PipeView& V, int ci, int cj) {
    const int h = V.R / 2;
    return ci > h + 1 && cj > h + 1 && ci < V.SX - h - 1 && cj < V.SY - h - 1;
}

__device__ inline double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ inline double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// getAandB's sums over the patch at `corner`, by one warp: *A of the pixels whose library
// PSF is not under thr and *B of those under it, pixel after pixel in the order of getAandB's
// loop (the even lanes add up B and the odd ones A); returns the number under thr.
__device__ int pipe_sums(const PipeView& V, const double* img, const double* psf, size_t corner, double thr, double* A,
                         double* B) {
    const double* vm = V.vmap;
    const int R = V.R, RR = R * R, SY = V.SY, lane = threadIdx.x & 31;
    auto pixel = [&](int k, bool& low) {
        if (k >= RR) return 0.0;
        const size_t px = corner + (size_t)(k / R) * SY + k % R;
        low = psf[k] < thr;
        return img[px] - (vm ? vm[px] : 0.0);
    };
    bool low = false;
    double v = pixel(lane, low), sum = 0;
    int cb = 0;
    for (int k0 = 0; k0 < RR; k0 += 32) {
        const unsigned lows = __ballot_sync(0xffffffffu, low);
        const double cur = v;
        low = false;
        v = pixel(k0 + 32 + lane, low);  // on its way while this one is added up
        const unsigned mine = (lane & 1) ? ~lows : lows;
        cb += __popc(lows);
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            const double x = __shfl_sync(0xffffffffu, cur, q);
            sum += (mine >> q & 1u) ? x : 0.0;
        }
    }
    *B = __shfl_sync(0xffffffffu, sum, 0);
    *A = __shfl_sync(0xffffffffu, sum, 1);
    return cb;
}

// Whether a candidate is fitted (maxPatch / B > maxSNR and B > 0), by one warp, with B
// of getAandB: the mean of the pixels whose library PSF of slice r is under 10% of its
// maximum, of the patch minus the sCMOS term when there is one (:1119-1211).  The lanes'
// own sums decide wherever the rounding of any order of the sum leaves no doubt (a sum of
// n terms is off by at most n u times the sum of their magnitudes), and pipe_sums else.
__device__ bool pipe_fitted(const PipeView& V, const double* img, int r, int ci, int cj, double* maxp_) {
    const double* vm = V.vmap;
    const int R = V.R, RR = R * R, SY = V.SY, lane = threadIdx.x & 31;
    const size_t corner = (size_t)(ci - R / 2) * SY + (cj - R / 2);
    const double* psf = V.libpsf + (size_t)r * RR;
    double maxp = -INFINITY, maxi = -INFINITY;
#pragma unroll 4
    for (int k = lane; k < RR; k += 32) {
        const size_t px = corner + (size_t)(k / R) * SY + k % R;
        maxi = fmax(maxi, psf[k]);
        maxp = fmax(maxp, img[px] - (vm ? vm[px] : 0.0));
    }
    maxi = warp_max(maxi);
    maxp = warp_max(maxp);
    const double thr = maxi * 0.1;
    double B = 0, mag = 0;
    int cb = 0;
#pragma unroll 4
    for (int k = lane; k < RR; k += 32) {
        const size_t px = corner + (size_t)(k / R) * SY + k % R;
        const bool low = psf[k] < thr;
        const double x = low ? img[px] - (vm ? vm[px] : 0.0) : 0.0;
        B += x;
        mag += fabs(x);
        cb += low;
    }
    B = warp_sum(B);
    mag = warp_sum(mag);
    cb = __reduce_add_sync(0xffffffffu, cb);
    *maxp_ = maxp;
    auto fitted = [&](double b) { return maxp / b > V.max_snr && b > 0; };
    if (cb == 0) return fitted(0.0);
    // both orders' sums and the roundings of the mean and the ratio, with room to spare; the
    // test is monotone in b on either side of zero
    const double err = 4e-16 * (RR + 8) * mag / cb, lo = B / cb - err, hi = B / cb + err;
    const double s_lo = V.max_snr * (1 - 1e-15), s_hi = V.max_snr * (1 + 1e-15);
    if (hi <= 0) return false;
    if (lo > 0) {
        const double a = maxp / lo, b = maxp / hi;
        if (fmin(a, b) > fmax(s_lo, s_hi)) return true;
        if (fmax(a, b) < fmin(s_lo, s_hi)) return false;
    }
    double A;
    pipe_sums(V, img, psf, corner, thr, &A, &B);
    return fitted(B / cb);
}

// near_mask from the mask, 32 rows of a frame a CTA: rows as words of bits, each the OR of
// its R neighbours along the row, then of R rows.  Most of a list's candidates lie near a
// mask late in a frame, and k_pipe_wave drops them by one bit (47 us a wave for 96 frames
// of 256^2 at R = 40); looking through their patches, a warp each, was 540 of its 630 us.
constexpr int PN_ROWS = 32, PN_THREADS = 256;
static size_t near_smem(int SY, int R) { return (size_t)2 * (PN_ROWS + R - 1) * ((SY + 31) / 32) * sizeof(unsigned); }
__global__ void __launch_bounds__(PN_THREADS) k_pipe_near(PipeView V) {
    extern __shared__ unsigned pn_sm[];
    const int f = blockIdx.y, SX = V.SX, SY = V.SY, R = V.R, h = R / 2, i0 = blockIdx.x * PN_ROWS;
    if (V.done[f]) return;
    const int WY = (SY + 31) / 32, rows = PN_ROWS + R - 1, lane = threadIdx.x & 31;
    unsigned *raw = pn_sm, *wide = raw + rows * WY;
    const unsigned char* mk = V.mask + (size_t)f * SX * SY;
#pragma unroll 4
    for (int q = threadIdx.x >> 5; q < rows * WY; q += PN_THREADS / 32) {
        const int i = i0 - h + q / WY, j = q % WY * 32 + lane;
        const unsigned b = __ballot_sync(0xffffffffu, i >= 0 && i < SX && j < SY && mk[(size_t)i * SY + j] != 0);
        if (lane == 0) raw[q] = b;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < rows * WY; q += PN_THREADS) {
        const int w = q % WY;
        const unsigned* row = raw + q - w;
        unsigned any = 0;
        for (int d = -h; d < R - h; ++d) {  // the 32 bits from bit 32 w + d on
            const int a = w + (d >> 5);
            const unsigned lo = a >= 0 && a < WY ? row[a] : 0, hi = a + 1 >= 0 && a + 1 < WY ? row[a + 1] : 0;
            any |= __funnelshift_r(lo, hi, d & 31);
        }
        wide[q] = any;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < PN_ROWS * WY; q += PN_THREADS) {
        if (i0 + q / WY >= SX) continue;
        unsigned any = 0;
        for (int d = 0; d < R; ++d) any |= wide[q + d * WY];
        V.near_mask[((size_t)f * SX + i0) * WY + q] = any;
    }
}

// One wave's selection for one frame (one CTA): walking the candidates from the
// frame's pointer, the first K (in candidate order) that need a fit under the
// current mask get slots and their ROI (k_pipe_start adds the start).  limit = just
// past the K-th (or the end).
// 512 candidates at a time: a thread drops the ones outside the border or with a masked
// pixel in their patch, which late in a frame are nearly all; the rest are taken in
// order, a warp each, until K are found: 90 us a wave at R = 40.  (A thread a candidate
// for everything read its 1,600 pixels one after the other: 2.8 ms.)
constexpr int PW_THREADS = 512, PW_WARPS = PW_THREADS / 32;
__global__ void __launch_bounds__(PW_THREADS) k_pipe_wave(PipeView V, int K) {
    const int f = blockIdx.x, SX = V.SX, SY = V.SY, R = V.R, h = R / 2, RR = R * R;
    if (V.done[f]) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double* img = V.fimg + (size_t)f * SX * SY;
    const unsigned* near_mask = V.near_mask + (size_t)f * SX * ((SY + 31) / 32);
    const double* cand = V.cand + (size_t)f * V.cap * 7;
    int* code_of = V.cand_slot + (size_t)f * V.cap;
    const int n = min(V.counts[f], V.cap);
    __shared__ int live[PW_THREADS], wcount[PW_WARPS], sel[PW_WARPS], s_base;
    int taken = 0, limit = n;
    for (int c0 = V.pointer[f]; c0 < n && taken < K; c0 += PW_THREADS) {
        const int i = c0 + threadIdx.x;
        bool look = false;
        if (i < n) {
            const int ci = (int)llrint(cand[(size_t)i * 7 + 2]), cj = (int)llrint(cand[(size_t)i * 7 + 3]);
            const bool in = pipe_inside(V, ci, cj);
            look = in && !(near_mask[(size_t)ci * ((SY + 31) / 32) + (cj >> 5)] >> (cj & 31) & 1u);
            if (!look) code_of[i] = in ? -3 : -2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, look);
        if (lane == 0) wcount[warp] = __popc(bal);
        __syncthreads();
        int at = 0, nl = 0;
        for (int w = 0; w < PW_WARPS; ++w) {
            if (w < warp) at += wcount[w];
            nl += wcount[w];
        }
        if (look) live[at + __popc(bal & ((1u << lane) - 1))] = i;
        __syncthreads();
        for (int l0 = 0; l0 < nl && taken < K; l0 += PW_WARPS) {
            const bool mine = l0 + warp < nl;
            const int k = live[min(l0 + warp, nl - 1)];
            const double* row = cand + (size_t)k * 7;
            const int r = (int)llrint(row[1]), ci = (int)llrint(row[2]), cj = (int)llrint(row[3]);
            const size_t corner = (size_t)(ci - h) * SY + (cj - h);
            double maxp = 0;
            int code = -3;
            if (mine) {
                code = pipe_fitted(V, img, r, ci, cj, &maxp) ? 0 : -1;
                if (lane == 0) {
                    code_of[k] = code;
                    V.cand_maxp[(size_t)f * V.cap + k] = maxp;
                }
            }
            if (lane == 0) sel[warp] = mine && code == 0;
            __syncthreads();
            int rank = 0, got = 0, last = -1;
            for (int w = 0; w < PW_WARPS; ++w)
                if (sel[w] && got < K - taken) {
                    if (w < warp) ++rank;
                    ++got;
                    last = w;
                }
            if (threadIdx.x == 0) s_base = got ? atomicAdd(V.nslots, got) : 0;
            __syncthreads();
            if (mine && code == 0 && warp <= last) {
                const int s = s_base + rank;
                if (lane == 0) code_of[k] = s < V.slot_cap ? s : -5;
                if (s < V.slot_cap) {
                    float* roi = V.rois + (size_t)s * RR;
                    float* sv = V.vmap ? V.slot_v + (size_t)s * RR : nullptr;
#pragma unroll 4
                    for (int q = lane; q < RR; q += 32) {
                        const size_t px = corner + (size_t)(q / R) * SY + q % R;
                        roi[q] = (float)img[px];
                        if (sv) sv[q] = (float)V.vmap[px];
                    }
                    if (lane == 0) {
                        V.slot_frame[s] = f;
                        V.slot_cand[s] = k;
                    }
                }
            }
            taken += got;
            if (taken == K) limit = live[l0 + last] + 1;
            __syncthreads();  // sel, s_base and live are written again
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) V.limit[f] = limit;
}

// Starts of the wave's slots: the candidates' refined offsets, loc.init(A, B, -dx, -dy,
// range[r] + dz), and getAandB's A and B.  A warp a slot: a split fit's path depends on the
// last bit of its start, so the sums keep the order of getAandB's loop.  (40 px: 1,600 adds,
// one after the other, about 30 us for a wave of 768 slots.)
__global__ void __launch_bounds__(128) k_pipe_start(PipeView V, int n) {
    const int s = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (s >= n) return;
    const double* row = V.cand + ((size_t)V.slot_frame[s] * V.cap + V.slot_cand[s]) * 7;
    const int R = V.R, RR = R * R;
    const int r = (int)llrint(row[1]), ci = (int)llrint(row[2]), cj = (int)llrint(row[3]);
    const double* img = V.fimg + (size_t)V.slot_frame[s] * V.SX * V.SY;
    const double* psf = V.libpsf + (size_t)r * RR;
    double maxi = -INFINITY;
#pragma unroll 4
    for (int k = lane; k < RR; k += 32) maxi = fmax(maxi, psf[k]);
    double A, B;
    const int cb = pipe_sums(V, img, psf, (size_t)(ci - R / 2) * V.SY + (cj - R / 2), warp_max(maxi) * 0.1, &A, &B);
    if (lane != 0) return;
    B = cb != 0 ? B / cb : 0.0;
    A -= (double)(RR - cb) * B;
    double* in = V.init + (size_t)s * 5;
    in[0] = -row[5];
    in[1] = -row[6];
    in[2] = V.range[r] + row[4];
    in[3] = A;
    in[4] = B;
}

// The fitted slots that can be accepted whatever the mask: every test of the
// walk's acceptance (k_pipe_replay) but the mask's, with the same arithmetic.
// Only these need the model at their fit (the walk masks by the model only
// where it accepts); they are listed in list[0 .. *count).
__device__ __forceinline__ bool pipe_static_pass(const PipeView& V, const double* theta, const int* status, int slot,
                                                 int ci, int cj) {
    if (status[slot] == ZOLA_FIT_NAN) return false;
    const double* th = theta + (size_t)slot * 5;
    const double x = th[0], y = th[1], z = th[2], A = th[3];
    if (!(A > V.photon_thr && fabs(x) < 10 * V.dx && fabs(y) < 10 * V.dx)) return false;
    const int px = (int)(ci - x / V.dx), py = (int)(cj - y / V.dx);
    return px >= 0 && px < V.SX && py >= 0 && py < V.SY && z > V.minZ && z < V.maxZ;
}

__global__ void k_pipe_need(PipeView V, int n, const double* theta, const int* status, int* list, int* count) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double* row = V.cand + ((size_t)V.slot_frame[s] * V.cap + V.slot_cand[s]) * 7;
    if (pipe_static_pass(V, theta, status, s, (int)llrint(row[2]), (int)llrint(row[3]))) list[atomicAdd(count, 1)] = s;
}

// Model threshold of each listed slot: 0.2 max(0, max(model - B)), model =
// psi A + B (+ sCMOS v) (maxModelThreshold, LocalizationPipeline.java:860-880).
// A warp a slot.
__global__ void __launch_bounds__(128) k_pipe_mthr(int n, int RR, const double* theta, const double* psi,
                                                   const float* slot_v, double* mthr, const int* list, const int* count) {
    const int li = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (li >= min(n, *count)) return;
    const int s = list[li];
    const double A = theta[5 * s + 3], B = theta[5 * s + 4];
    const double* ps = psi + (size_t)s * RR;
    const float* sv = slot_v ? slot_v + (size_t)s * RR : nullptr;
    double m = 0.0;
#pragma unroll 4
    for (int k = lane; k < RR; k += 32) m = fmax(m, ps[k] * A + B + (sv ? (double)sv[k] : 0.0) - B);
    m = warp_max(m);
    if (lane == 0) mthr[s] = m * 0.2;
}

// The reference's sequential walk over one frame's candidates (one CTA per
// frame), with the speculative fits.  Accepted slots are listed with their
// candidate index as the in-frame order.
__global__ void __launch_bounds__(256) k_pipe_replay(PipeView V, const double* theta, const int* status,
                                                     const double* psi, const double* mthr, int* acc_slot,
                                                     int* acc_seq, int* nacc) {
    const int f = blockIdx.x, SX = V.SX, SY = V.SY, R = V.R, h = R / 2, RR = R * R;
    unsigned char* mk = V.mask + (size_t)f * SX * SY;
    const double* img = V.fimg + (size_t)f * SX * SY;
    const double* cand = V.cand + (size_t)f * V.cap * 7;
    if (V.done[f]) return;
    const int n = min(V.counts[f], V.cap), lim = V.limit[f], warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The candidates to walk, in order: 256 at a time, without those outside the border
    // or already masked when the wave looked (masks only grow).
    __shared__ int list[256], wcount[8];
    int c0 = V.pointer[f] - 256, at = 0, nl = 0;
    for (;;) {
        if (at == nl) {
            c0 += 256;
            if (c0 >= lim) break;
            __syncthreads();
            const int k = c0 + threadIdx.x, code = k < lim ? V.cand_slot[(size_t)f * V.cap + k] : -2;
            const unsigned bal = __ballot_sync(0xffffffffu, code != -2 && code != -3);
            if (lane == 0) wcount[warp] = __popc(bal);
            __syncthreads();
            int o = at = nl = 0;
            for (int w = 0; w < 8; ++w) {
                if (w < warp) o += wcount[w];
                nl += wcount[w];
            }
            if (code != -2 && code != -3) list[o + __popc(bal & ((1u << lane) - 1))] = k;
            __syncthreads();
            continue;
        }
        const int i = list[at++], slot = V.cand_slot[(size_t)f * V.cap + i];
        const int ci = (int)llrint(cand[(size_t)i * 7 + 2]), cj = (int)llrint(cand[(size_t)i * 7 + 3]);
        if (mk[(size_t)ci * SY + cj]) continue;  // uniform read of the (synchronised) mask
        bool mine = false;
        for (int k = threadIdx.x; k < RR; k += blockDim.x)
            mine |= mk[(size_t)(ci - h + k / R) * SY + (cj - h + k % R)] != 0;
        if (__syncthreads_or(mine)) continue;  // alreadyTreated
        const double maxp = V.cand_maxp[(size_t)f * V.cap + i];
        bool accepted = false;
        if (slot >= 0 && pipe_static_pass(V, theta, status, slot, ci, cj)) {
            const double* th = theta + (size_t)slot * 5;
            const int px = (int)(ci - th[0] / V.dx), py = (int)(cj - th[1] / V.dx);
            accepted = !mk[(size_t)px * SY + py];
        }
        __syncthreads();  // every thread has read the mask before it changes
        if (accepted) {
            if (threadIdx.x == 0) {
                const int o = atomicAdd(nacc, 1);
                acc_slot[o] = slot;
                acc_seq[o] = i;
            }
            const double A = theta[(size_t)slot * 5 + 3], B = theta[(size_t)slot * 5 + 4], thr = mthr[slot];
            const double* ps = psi + (size_t)slot * RR;
            const float* sv = V.vmap ? V.slot_v + (size_t)slot * RR : nullptr;
            for (int k = threadIdx.x; k < RR; k += blockDim.x)
                if (ps[k] * A + B + (sv ? (double)sv[k] : 0.0) - B > thr)
                    mk[(size_t)(ci - h + k / R) * SY + (cj - h + k % R)] = 1;
        } else {
            for (int k = threadIdx.x; k < RR; k += blockDim.x) {
                const size_t px = (size_t)(ci - h + k / R) * SY + (cj - h + k % R);
                if (img[px] > maxp * 0.5) mk[px] = 1;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        V.pointer[f] = lim;
        V.done[f] = lim >= n;
    }
}

struct LocRow {
    int frame, seq, status;
    double x, y, z, A, B, chi2, cx, cy, cz;
};

__global__ void k_take_xyz(int n, const double* theta, double* xyz) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n)
        for (int q = 0; q < 3; ++q) xyz[3 * s + q] = theta[5 * (size_t)s + q];
}

__global__ void k_take_acc(int n, const int* acc_slot, const double* theta, double* xyz) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n)
        for (int q = 0; q < 3; ++q) xyz[3 * k + q] = theta[5 * (size_t)acc_slot[k] + q];
}

// chi2 and CRLB of the accepted localizations (psi, dpsi evaluated at their
// fitted positions by direct sums, in acceptance-list order: at z = 0 of a PSF that is the
// same above and below focus the z bound is made of the derivatives' last bits).  A warp a row; a thread a row read
// its 4 R^2 model values one after the other (2.0 ms for 100 rows at R = 40).
__global__ void __launch_bounds__(128) k_pipe_rows(PipeView V, int n, const int* acc_slot, const int* acc_seq,
                                                   const int* status, const double* theta, const double* psi,
                                                   const double* dpsi, LocRow* rows) {
    const int k = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= n) return;
    const int s = acc_slot[k], R = V.R, RR = R * R;
    const int f = V.slot_frame[s], i = V.slot_cand[s];
    const double* row = V.cand + ((size_t)f * V.cap + i) * 7;
    const int ci = (int)llrint(row[2]), cj = (int)llrint(row[3]);
    const double* th = theta + (size_t)s * 5;
    const double x = th[0], y = th[1], z = th[2], A = th[3], B = th[4];
    const double* ps = psi + (size_t)k * RR;
    const float* roi = V.rois + (size_t)s * RR;
    const float* sv = V.vmap ? V.slot_v + (size_t)s * RR : nullptr;
    double chi = 0, acc[15];
#pragma unroll
    for (int q = 0; q < 15; ++q) acc[q] = 0;
#pragma unroll 2
    for (int p = lane; p < RR; p += 32) {
        const double m = ps[p] * A + B, mu = m + (sv ? (double)sv[p] : 0.0);
        const double dd = roi[p] - mu;  // scoreCompute against the model (with the sCMOS term)
        chi += dd * dd / mu;
        const double d[5] = {A * dpsi[((size_t)k * 3 + 0) * RR + p], A * dpsi[((size_t)k * 3 + 1) * RR + p],
                             A * dpsi[((size_t)k * 3 + 2) * RR + p], m, 1.0};
        int o = 0;
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
            for (int r2 = 0; r2 <= q; ++r2) acc[o++] += d[q] * d[r2] / m;
    }
    chi = warp_sum(chi) / RR;
#pragma unroll
    for (int q = 0; q < 15; ++q) acc[q] = warp_sum(acc[q]);
    if (lane != 0) return;
    double F[25];
    int o = 0;
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int r2 = 0; r2 <= q; ++r2) F[q * 5 + r2] = F[r2 * 5 + q] = acc[o++];
    double cr[5];
    lm_crlb(F, cr);
    for (int q = 0; q < 3; ++q)
        if (!(cr[q] == cr[q])) cr[q] = F[q * 5 + q] != 0 ? sqrt(1.0 / F[q * 5 + q]) : 1.79769313486231570e308;
    LocRow& L = rows[k];
    L.frame = f; L.seq = acc_seq[k]; L.status = status[s];
    L.x = 1000 * (ci * V.dx - x); L.y = 1000 * (cj * V.dx - y); L.z = 1000 * z;
    L.A = A; L.B = B; L.chi2 = chi;
    L.cx = 1000 * cr[0]; L.cy = 1000 * cr[1]; L.cz = 1000 * cr[2];
}

}  // namespace zola

using namespace zola;

namespace {

struct Buf {
    void* p = nullptr;
    size_t bytes = 0;
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    ~Buf() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t b) {
        if (b <= bytes && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, b ? b : 1);
        if (e == cudaSuccess) bytes = b ? b : 1;
        return e;
    }
};

// Speculative fits per frame and wave: 8, and up to 64 in split fits of few frames.  A round
// of a split fit costs nearly the same until every SM has a unit or two (4 slots for 3 SMs
// at a window of 128, 4 an SM at 64, 10 at 32), and more fits a wave make fewer waves; beyond
// that, the fits of candidates that an acceptance of the same wave masks are not free.
// At 8 and at this rule's (148 SMs): 2 frames of 40 px 42 and 21 ms, 12 of them 56 and 46, 6 of 24 px
// 56 and 30, 20 of 16 px 35 and 18; 96 frames of 40 px at 8, 12 and 16: 146, 160 and 176.
constexpr int PIPE_WAVE_FITS = 8, PIPE_WAVE_MAX = 64;
int wave_fits(int sms, int R, int N, int frames, int precision) {
    if (precision != ZOLA_PREC_SPLIT) return PIPE_WAVE_FITS;
    const int W = window_size(R, N), slots = W >= 128 ? 4 * sms / 3 : W >= 64 ? 4 * sms : 10 * sms;
    return std::max(PIPE_WAVE_FITS, std::min(PIPE_WAVE_MAX, slots / frames));
}
// Candidates stored per frame at the start of a call: a 256 x 256 frame against a
// 41-slice library lists up to about 7,500 at the reference's threshold.
constexpr int PIPE_CAND_ROOM = 8192;

}  // namespace

namespace zola {

// sCMOS frames (LocalizationPipeline.java:588-640): c = (ADU - offset)/gain;
// detection image c + vargain[0] clamped at 0, fit image c + vargain.
__global__ void k_pipe_scmos(const float* adu, const double* offset, const double* gain, const double* vg, size_t SS,
                             int nf, double* det_img, double* fit_img) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < SS * nf; k += (size_t)gridDim.x * blockDim.x) {
        const size_t px = k % SS;
        const double c = ((double)adu[k] - offset[px]) / gain[px];
        const double d = c + vg[0];
        det_img[k] = d < 0 ? 0 : d;
        fit_img[k] = c + vg[px];
    }
}

}  // namespace zola

namespace {

// frames: photon frames (no sCMOS); or adu + offset/gain/variance maps (sCMOS).
// u16: camera counts (with rescale = {slope, intercept}) instead of photon frames.
int localize_impl(zola_ctx* ctx, zola_detector* det, zola_psf* fit_psf, const double* frames, const float* adu,
                  const double* offset, const double* gain, const double* variance, int nframes, int frame0,
                  const zola_loc_params* prm, zola_localization* out, int out_cap, int* nout,
                  const uint16_t* u16 = nullptr, const double* rescale = nullptr) {
    const bool scmos = adu != nullptr;
    *nout = 0;
    if (nframes <= 0) return ZOLA_OK;
    const int SX = det->v.SX, SY = det->v.SY, R = det->v.R;
    if (det->psf->ctx != ctx || fit_psf->ctx != ctx) { ctx->err = "zola_localize_frames: objects of another context"; return ZOLA_E_ARG; }
    if (prm->patch != R) { ctx->err = "zola_localize_frames: params.patch must equal the detector's R"; return ZOLA_E_ARG; }
    if (fit_psf->o.kz_reset) { ctx->err = "zola_localize_frames: the fit PSF needs kz_reset = 0"; return ZOLA_E_ARG; }
    const std::vector<double>& range = det->range;
    const std::vector<double>& lib = det->h_psf;
    // candidates stored per frame: grows to the longest list met, so that every
    // frame walks its whole list as the reference does
    int cap = prm->cand_cap > 0 ? prm->cand_cap : std::max(PIPE_CAND_ROOM, det->cand_room);
    if (cap > ZOLA_DETECT_MAX_CAP) { ctx->err = "zola_localize_frames: cand_cap above 2^20"; return ZOLA_E_ARG; }
    const int FB = std::max(1, std::min(nframes, prm->frames_per_batch > 0 ? prm->frames_per_batch : 1024));
    const size_t SS = (size_t)SX * SY, RR = (size_t)R * R;
    cudaStream_t st = ctx->stream;
    ZOLA_CUDA_CHECK(cudaFuncSetAttribute(k_pipe_near, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)near_smem(SY, R)),
                    ctx);
    const int K = prm->wave_fits > 0 ? prm->wave_fits : wave_fits(ctx->num_sms, R, fit_psf->N, FB, prm->precision);
    const int slot_cap = FB * K;
    Buf b_img, b_mask, b_cand, b_cnt, b_lib, b_rng, b_cslot, b_cmax, b_ptr, b_lim, b_done, b_ns, b_rois, b_init, b_sf,
        b_sc, b_out5, b_st, b_xyz, b_psi, b_mthr, b_acc, b_seq, b_nacc, b_dpsi, b_rows, b_fimg, b_adu, b_off, b_gain,
        b_vg, b_sv, b_u16, b_list, b_nlist, b_var, b_near;
    cudaError_t e = cudaSuccess;
    auto A = [&](Buf& b, size_t bytes) { if (e == cudaSuccess) e = b.alloc(bytes); };
    A(b_img, SS * FB * 8); A(b_var, SS * FB * 8); A(b_mask, SS * FB); A(b_near, (size_t)FB * SX * ((SY + 31) / 32) * 4); A(b_cand, (size_t)FB * cap * 7 * 8); A(b_cnt, (size_t)FB * 4);
    A(b_lib, lib.size() * 8); A(b_rng, range.size() * 8); A(b_cslot, (size_t)FB * cap * 4);
    A(b_cmax, (size_t)FB * cap * 8); A(b_ptr, (size_t)FB * 4); A(b_lim, (size_t)FB * 4); A(b_done, (size_t)FB * 4);
    A(b_ns, 64); A(b_nacc, 64);
    A(b_rois, RR * slot_cap * 4); A(b_init, (size_t)slot_cap * 40); A(b_sf, (size_t)slot_cap * 4);
    A(b_sc, (size_t)slot_cap * 4); A(b_out5, (size_t)slot_cap * 40); A(b_st, (size_t)slot_cap * 4);
    A(b_xyz, (size_t)slot_cap * 24); A(b_psi, RR * slot_cap * 8); A(b_mthr, (size_t)slot_cap * 8);
    A(b_acc, (size_t)slot_cap * 4); A(b_seq, (size_t)slot_cap * 4);
    if (u16) A(b_u16, SS * FB * 2);
    A(b_list, (size_t)slot_cap * 4); A(b_nlist, 64);
    if (scmos) {
        A(b_fimg, SS * FB * 8); A(b_adu, SS * FB * 4); A(b_off, SS * 8); A(b_gain, SS * 8); A(b_vg, SS * 8);
        A(b_sv, RR * slot_cap * 4);
        std::vector<double> vg(SS);
        for (size_t k = 0; k < SS; ++k) vg[k] = variance[k] / (gain[k] * gain[k]);  // SCMOScamera.java:95
        if (e == cudaSuccess) e = cudaMemcpy(b_vg.p, vg.data(), SS * 8, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(b_off.p, offset, SS * 8, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(b_gain.p, gain, SS * 8, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(b_lib.p, lib.data(), lib.size() * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b_rng.p, range.data(), range.size() * 8, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) { ctx->err = std::string("zola_localize_frames: ") + cudaGetErrorString(e); return ZOLA_E_CUDA; }
    zola_fit_params fp{prm->minZ - 0.3, prm->maxZ + 0.3, 10 * fit_psf->o.xystep + 1e-3, prm->max_iter, prm->tol_xyz,
                       fit_psf->o.xystep, 2 * fit_psf->o.xystep, prm->precision};
    PipeView V{};
    V.SX = SX; V.SY = SY; V.R = R; V.cap = cap;
    V.dx = fit_psf->o.xystep; V.minZ = prm->minZ; V.maxZ = prm->maxZ; V.photon_thr = prm->photon_threshold;
    V.max_snr = prm->max_snr;
    V.images = (double*)b_img.p; V.mask = (unsigned char*)b_mask.p; V.near_mask = (unsigned*)b_near.p; V.cand = (double*)b_cand.p;
    V.fimg = scmos ? (double*)b_fimg.p : (double*)b_img.p;
    V.vmap = scmos ? (double*)b_vg.p : nullptr;
    V.slot_v = scmos ? (float*)b_sv.p : nullptr;
    V.counts = (int*)b_cnt.p; V.libpsf = (double*)b_lib.p; V.range = (double*)b_rng.p;
    V.cand_slot = (int*)b_cslot.p; V.cand_maxp = (double*)b_cmax.p; V.pointer = (int*)b_ptr.p;
    V.limit = (int*)b_lim.p; V.done = (int*)b_done.p; V.nslots = (int*)b_ns.p; V.slot_cap = slot_cap;
    V.rois = (float*)b_rois.p; V.init = (double*)b_init.p; V.slot_frame = (int*)b_sf.p; V.slot_cand = (int*)b_sc.p;
    std::vector<LocRow> all;
    std::vector<int> done;
    auto fail = [&](cudaError_t err) {
        ctx->err = std::string("zola_localize_frames: ") + cudaGetErrorString(err);
        return ZOLA_E_CUDA;
    };
    for (int f0 = 0; f0 < nframes; f0 += FB) {
        const int nf = std::min(FB, nframes - f0);
        V.nframes = nf;
        if (scmos) {
            e = copy_in(ctx, b_adu.p, adu + (size_t)f0 * SS, SS * nf * 4, st);
            if (e == cudaSuccess) {
                k_pipe_scmos<<<ctx->num_sms * 8, 256, 0, st>>>((float*)b_adu.p, (double*)b_off.p, (double*)b_gain.p,
                                                              (double*)b_vg.p, SS, nf, (double*)b_img.p,
                                                              (double*)b_fimg.p);
                ctx->launches++;
            }
        } else if (u16) {  // 2 bytes a pixel over the host link, photons made on the device
            e = copy_in(ctx, b_u16.p, u16 + (size_t)f0 * SS, SS * nf * 2, st);
            if (e == cudaSuccess) rescale_u16(ctx, (const uint16_t*)b_u16.p, SS * nf, rescale, (double*)b_img.p, st);
        } else {
            e = copy_in(ctx, b_img.p, frames + (size_t)f0 * SS, SS * nf * 8, st);
        }
        if (e == cudaSuccess) e = cudaMemsetAsync(b_mask.p, 0, SS * nf, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(b_ptr.p, 0, (size_t)nf * 4, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(b_done.p, 0, (size_t)nf * 4, st);
        if (e != cudaSuccess) return fail(e);
        // positions and order of every candidate; the offsets of those that get a fit follow per wave
        int rc = detect_frames(det, (double*)b_img.p, nf, cap, cap, 0, (double*)b_cand.p, (int*)b_cnt.p,
                               (double*)b_var.p, st);
        if (rc) return rc;
        std::vector<int> counts(nf);
        e = cudaMemcpyAsync(counts.data(), b_cnt.p, (size_t)nf * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return fail(e);
        const int longest = *std::max_element(counts.begin(), counts.end());
        det->cand_room = std::max(det->cand_room, longest);
        if (longest > cap) {  // room for every candidate; the frames whose list was cut are detected again
            if (longest > ZOLA_DETECT_MAX_CAP) {
                ctx->err = "zola_localize_frames: a frame has more than 2^20 candidates";
                return ZOLA_E_ARG;
            }
            const int old = cap;
            cap = longest;
            {
                // the stored rows move to the wider layout; the frames whose whole list
                // fitted keep them (detection is per frame, so they would come out the same)
                Buf wide;
                e = wide.alloc((size_t)FB * cap * 7 * 8);
                if (e == cudaSuccess)
                    e = cudaMemcpy2DAsync(wide.p, (size_t)cap * 7 * 8, b_cand.p, (size_t)old * 7 * 8,
                                          (size_t)old * 7 * 8, nf, cudaMemcpyDeviceToDevice, st);
                if (e != cudaSuccess) return fail(e);
                std::swap(b_cand.p, wide.p);
                std::swap(b_cand.bytes, wide.bytes);
            }  // (freeing the old rows waits for the copy)
            A(b_cslot, (size_t)FB * cap * 4); A(b_cmax, (size_t)FB * cap * 8);
            if (e != cudaSuccess) return fail(e);
            V.cap = cap;
            V.cand = (double*)b_cand.p; V.cand_slot = (int*)b_cslot.p; V.cand_maxp = (double*)b_cmax.p;
            // the cut frames, gathered, are detected again as one batch and their rows scattered back
            std::vector<int> cut;
            for (int f = 0; f < nf; ++f)
                if (counts[f] > old) cut.push_back(f);
            const size_t nc = cut.size();
            Buf g_img, g_out, g_cnt;
            e = g_img.alloc(nc * SS * 8);
            if (e == cudaSuccess) e = g_out.alloc(nc * (size_t)cap * 7 * 8);
            if (e == cudaSuccess) e = g_cnt.alloc(nc * 4);
            for (size_t k = 0; k < nc && e == cudaSuccess; ++k)
                e = cudaMemcpyAsync((double*)g_img.p + k * SS, (double*)b_img.p + (size_t)cut[k] * SS, SS * 8,
                                    cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) return fail(e);
            rc = detect_frames(det, (double*)g_img.p, (int)nc, cap, cap, 0, (double*)g_out.p, (int*)g_cnt.p, nullptr, st);
            if (rc) return rc;
            for (size_t k = 0; k < nc && e == cudaSuccess; ++k) {
                e = cudaMemcpyAsync((double*)b_cand.p + (size_t)cut[k] * cap * 7, (double*)g_out.p + k * cap * 7,
                                    (size_t)cap * 7 * 8, cudaMemcpyDeviceToDevice, st);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync((int*)b_cnt.p + cut[k], (int*)g_cnt.p + k, 4, cudaMemcpyDeviceToDevice, st);
            }
            if (e != cudaSuccess) return fail(e);
        }  // (freeing the gathered buffers waits for the copies)
        for (int wave = 0;; ++wave) {
            e = cudaMemsetAsync(b_ns.p, 0, 4, st);
            if (e == cudaSuccess) e = cudaMemsetAsync(b_nacc.p, 0, 4, st);
            if (e != cudaSuccess) return fail(e);
            k_pipe_near<<<dim3((SX + PN_ROWS - 1) / PN_ROWS, nf), PN_THREADS, near_smem(SY, R), st>>>(V);
            k_pipe_wave<<<nf, PW_THREADS, 0, st>>>(V, K);
            ctx->launches += 2;
            int nslot = 0;
            e = cudaMemcpyAsync(&nslot, b_ns.p, 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return fail(e);
            if (nslot > 0) {
                rc = detect_refine(det, (double*)b_img.p, (double*)b_var.p, (double*)b_cand.p, cap, nslot,
                                   (int*)b_sf.p, (int*)b_sc.p, st);
                if (rc) return rc;
                k_pipe_start<<<(nslot + 3) / 4, 128, 0, st>>>(V, nslot);
                ctx->launches++;
                rc = fit_frames_dev(ctx, fit_psf, R, (float*)b_rois.p, V.slot_v, (double*)b_init.p, nslot, &fp,
                                    (double*)b_out5.p, (int*)b_st.p, st);
                if (rc) return rc;
                // psi at the fitted positions the walk may accept (its model masks)
                k_take_xyz<<<(nslot + 127) / 128, 128, 0, st>>>(nslot, (double*)b_out5.p, (double*)b_xyz.p);
                e = cudaMemsetAsync(b_nlist.p, 0, 4, st);
                if (e != cudaSuccess) return fail(e);
                k_pipe_need<<<(nslot + 127) / 128, 128, 0, st>>>(V, nslot, (double*)b_out5.p, (int*)b_st.p,
                                                                 (int*)b_list.p, (int*)b_nlist.p);
                ctx->launches += 2;
                WindowTables* wt = get_window(fit_psf, R, ctx->err);
                if (!wt) return ZOLA_E_ARG;
                rc = launch_model_f64(ctx, fit_psf, wt, (double*)b_xyz.p, nslot, (double*)b_psi.p, nullptr, st,
                                      (const int*)b_list.p, (const int*)b_nlist.p);
                if (rc) return rc;
                k_pipe_mthr<<<(nslot + 3) / 4, 128, 0, st>>>(nslot, (int)RR, (double*)b_out5.p,
                                                                 (double*)b_psi.p, V.slot_v, (double*)b_mthr.p,
                                                                 (const int*)b_list.p, (const int*)b_nlist.p);
                ctx->launches++;
            }
            k_pipe_replay<<<nf, 256, 0, st>>>(V, (double*)b_out5.p, (int*)b_st.p, (double*)b_psi.p,
                                             (double*)b_mthr.p, (int*)b_acc.p, (int*)b_seq.p, (int*)b_nacc.p);
            ctx->launches++;
            int nacc = 0;
            done.assign(nf, 0);
            e = cudaMemcpyAsync(&nacc, b_nacc.p, 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(done.data(), b_done.p, (size_t)nf * 4, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return fail(e);
            if (nacc > 0) {
                A(b_dpsi, 3 * RR * (size_t)nacc * 8); A(b_rows, (size_t)nacc * sizeof(LocRow));
                if (e != cudaSuccess) return fail(e);
                k_take_acc<<<(nacc + 127) / 128, 128, 0, st>>>(nacc, (int*)b_acc.p, (double*)b_out5.p,
                                                               (double*)b_xyz.p);
                ctx->launches++;
                // the walk has used psi; its buffer now takes the accepted positions' models
                WindowTables* wt = get_window(fit_psf, R, ctx->err);
                if (!wt) return ZOLA_E_ARG;
                rc = launch_model_direct(ctx, fit_psf, wt, (double*)b_xyz.p, nacc, (double*)b_psi.p, (double*)b_dpsi.p, st);
                if (rc) return rc;
                k_pipe_rows<<<(nacc + 3) / 4, 128, 0, st>>>(V, nacc, (int*)b_acc.p, (int*)b_seq.p, (int*)b_st.p,
                                                                (double*)b_out5.p, (double*)b_psi.p,
                                                                (double*)b_dpsi.p, (LocRow*)b_rows.p);
                ctx->launches++;
                std::vector<LocRow> rows(nacc);
                e = cudaMemcpyAsync(rows.data(), b_rows.p, (size_t)nacc * sizeof(LocRow), cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
                if (e != cudaSuccess) return fail(e);
                for (auto& r : rows) r.frame += f0;
                all.insert(all.end(), rows.begin(), rows.end());
            }
            if (std::all_of(done.begin(), done.end(), [](int d) { return d != 0; })) break;
        }
    }
    std::sort(all.begin(), all.end(), [](const LocRow& a, const LocRow& b) {
        return a.frame != b.frame ? a.frame < b.frame : a.seq < b.seq;
    });
    if ((int)all.size() > out_cap) { ctx->err = "zola_localize_frames: out_cap too small"; *nout = (int)all.size(); return ZOLA_E_ARG; }
    for (size_t k = 0; k < all.size(); ++k) {
        const LocRow& r = all[k];
        zola_localization& L = out[k];
        L.id = (int)k;
        L.frame = frame0 + r.frame;
        L.x_nm = r.x; L.y_nm = r.y; L.z_nm = r.z; L.intensity = r.A; L.background = r.B; L.chi2 = r.chi2;
        L.crlb_x_nm = r.cx; L.crlb_y_nm = r.cy; L.crlb_z_nm = r.cz;
        L.candidate = r.seq;
        L.fit_status = r.status;
    }
    *nout = (int)all.size();
    return ZOLA_OK;
}

}  // namespace

extern "C" int zola_localize_frames(zola_ctx* ctx, zola_detector* det, zola_psf* fit_psf, const double* frames,
                                    int nframes, int frame0, const zola_loc_params* prm, zola_localization* out,
                                    int out_cap, int* nout) {
    if (!ctx || !det || !fit_psf || !prm || !nout || (nframes > 0 && (!frames || !out))) return ZOLA_E_ARG;
    return localize_impl(ctx, det, fit_psf, frames, nullptr, nullptr, nullptr, nullptr, nframes, frame0, prm, out,
                         out_cap, nout);
}

extern "C" int zola_localize_frames_u16(zola_ctx* ctx, zola_detector* det, zola_psf* fit_psf, const uint16_t* frames,
                                        int nframes, int frame0, const zola_loc_params* prm, double adu, double gain,
                                        double offset, zola_localization* out, int out_cap, int* nout) {
    if (!ctx || !det || !fit_psf || !prm || !nout || (nframes > 0 && (!frames || !out))) return ZOLA_E_ARG;
    if (!(gain != 0) || !std::isfinite(adu) || !std::isfinite(gain) || !std::isfinite(offset)) {
        ctx->err = "zola_localize_frames_u16: adu, gain, offset must be finite and gain non-zero";
        return ZOLA_E_ARG;
    }
    double rescale[2];
    camera_rescale(adu, gain, offset, rescale);
    return localize_impl(ctx, det, fit_psf, nullptr, nullptr, nullptr, nullptr, nullptr, nframes, frame0, prm, out,
                         out_cap, nout, frames, rescale);
}

extern "C" int zola_localize_frames_scmos(zola_ctx* ctx, zola_detector* det, zola_psf* fit_psf, const float* adu,
                                          int nframes, int frame0, const zola_loc_params* prm, const double* offset,
                                          const double* gain, const double* variance, zola_localization* out,
                                          int out_cap, int* nout) {
    if (!ctx || !det || !fit_psf || !prm || !nout || (nframes > 0 && (!adu || !out)) || !offset || !gain || !variance)
        return ZOLA_E_ARG;
    return localize_impl(ctx, det, fit_psf, nullptr, adu, offset, gain, variance, nframes, frame0, prm, out, out_cap,
                         nout);
}

// ThunderStorm-style CSV (data/PLocalization.java:224-306): values floored to
// 1e-3 (PLocalization.java:59-72) and printed as Java's Double.toString does.
namespace {

std::string java_double(double v) {
    if (v != v) return "NaN";
    if (std::isinf(v)) return v > 0 ? "Infinity" : "-Infinity";
    if (v == 0) return std::signbit(v) ? "-0.0" : "0.0";
    char buf[64];
    int prec = 1;
    for (; prec <= 17; ++prec) {  // shortest round-trip digits
        std::snprintf(buf, sizeof buf, "%.*e", prec - 1, v);
        if (std::strtod(buf, nullptr) == v) break;
    }
    // buf = d.ddddde[+-]XX ; split into digits and exponent
    std::string s(buf);
    size_t epos = s.find('e');
    int exp10 = std::atoi(s.c_str() + epos + 1);
    std::string mant = s.substr(0, epos);
    bool neg = mant[0] == '-';
    if (neg) mant = mant.substr(1);
    std::string digits;
    for (char c : mant) if (c != '.') digits += c;
    while (digits.size() > 1 && digits.back() == '0') digits.pop_back();
    std::string r;
    const double a = std::fabs(v);
    if (a >= 1e-3 && a < 1e7) {
        int point = exp10 + 1;  // digits before the decimal point
        if (point <= 0) {
            r = "0." + std::string(-point, '0') + digits;
        } else if ((int)digits.size() <= point) {
            r = digits + std::string(point - digits.size(), '0') + ".0";
        } else {
            r = digits.substr(0, point) + "." + digits.substr(point);
        }
    } else {
        r = digits.substr(0, 1) + "." + (digits.size() > 1 ? digits.substr(1) : std::string("0")) + "E" +
            std::to_string(exp10);
    }
    return neg ? "-" + r : r;
}

double floor3(double v) { return std::floor(1000 * v) / 1000; }

}  // namespace

extern "C" int zola_write_csv(const char* path, const zola_localization* locs, int n, int append) {
    if (!path || n < 0 || (n > 0 && !locs)) return ZOLA_E_ARG;
    FILE* fp = std::fopen(path, append ? "a" : "w");
    if (!fp) return ZOLA_E_ARG;
    if (!append)
        std::fputs("id,frame,x [nm],y [nm],z [nm],intensity,background,chi2,crlbX,crlbY,crlbZ,driftX,driftY,driftZ,"
                   "occurrenceMerging\n", fp);
    for (int k = 0; k < n; ++k) {
        const zola_localization& L = locs[k];
        std::string line = std::to_string(L.id) + "," + std::to_string(L.frame) + "," + java_double(floor3(L.x_nm)) +
                           "," + java_double(floor3(L.y_nm)) + "," + java_double(floor3(L.z_nm)) + "," +
                           java_double(floor3(L.intensity)) + "," + java_double(floor3(L.background)) + "," +
                           java_double(floor3(L.chi2)) + "," + java_double(floor3(L.crlb_x_nm)) + "," +
                           java_double(floor3(L.crlb_y_nm)) + "," + java_double(floor3(L.crlb_z_nm)) +
                           ",0.0,0.0,0.0,1\n";
        std::fputs(line.c_str(), fp);
    }
    std::fclose(fp);
    return ZOLA_OK;
}

extern "C" int zola_format_double_java(double v, char* buf, int len) {
    if (!buf || len <= 0) return ZOLA_E_ARG;
    std::string s = java_double(v);
    if ((int)s.size() + 1 > len) return ZOLA_E_ARG;
    std::memcpy(buf, s.c_str(), s.size() + 1);
    return ZOLA_OK;
}
