// Correlation of camera frames with the detector's library through FP64 FFTs.
//
// The detector needs corr_r(i, j) = sum_uv img[i+u-R/2][j+v-R/2] psf0_r[u][v] for
// every library slice r.  The direct sum costs 2 S^2 R^2 Z flops a frame and is
// bound by the FP64 pipe (256^2 px, R = 40, 40 slices: 8.4 GFLOP, 310 us a frame
// at 27 TFLOP/s).  On an MX x MY grid with M >= S + R/2 the circular correlation
// equals it (both halos fall into the same zero padding), and costs about
// 0.2 GFLOP a frame: 30 us for that frame, 17 in the columns and 13 in the rows,
// which are bound by the L2 traffic and latency of T, the spectra and the scores
// (46 and 40 bytes a point; 18% of the FP64 rate).  These scores only screen the candidates: detect.cu takes
// its decisions with the error bound below, and computes the rows it returns by
// the direct sum.
//
// Two slices share one complex transform: with K = conj(FFT(p_r - i p_{r+1})),
// IFFT(FFT(img) K) holds corr_r in its real and corr_{r+1} in its imaginary part.
//   k_fft_rows_fwd   rows of the frames (or of the library pairs) -> A
//   k_fft_cols_fwd   columns of A -> spectra
//   k_fft_cols_inv   spectrum x K, inverse along columns -> T (rows 0 .. SX - 1)
//   k_fft_rows_inv   inverse along rows, scaled to scores, both slices written
// A line transform is a sequence of Stockham passes of radix 4, 5, 6 or 8.  TL
// neighbouring lines share a CTA and the lane index runs over the lines first, so
// every shared-memory access is conflict-free without padding, a warp reads only
// a few different twiddles, and every global sector is used whole.  A thread owns
// at most one butterfly a pass: its operands stay in registers over the barrier,
// and one in-place buffer suffices.  The first pass reads from global memory and
// the last one writes there, so a line of three passes crosses shared memory twice.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "fft_f64.h"
#include "zola_internal.h"

namespace zola {

// A line length M = R0 R1 R2 [R3] and how a CTA runs it, all known at compile
// time: radices behind a run-time switch put the operands in local memory and
// cost eight integer instructions to each floating-point one (57 and 69 us for
// the two inverse passes of two 256^2 frames, against 38 and 46 us at the time).
template <int R0, int R1, int R2, int R3>
struct Len {
    static constexpr int M = R0 * R1 * R2 * R3, NP = R3 > 1 ? 4 : 3;
    static constexpr int LEAST = R3 > 1 ? R3 : R2;  // radices come largest first
};

// A CTA's share: 1 << MOST lines, or fewer so that it has at most 400 threads (512 for
// two), and as many CTAs an SM as leave 56 registers a thread.  Columns are read and
// written along the lines and take 8; rows are read along the points, and the fewer
// lines the longer the runs: 2.  The inverse passes of two 256^2 frames take 33 + 27 us;
// rows with 4 lines and with 1 take 29 and 35, and with 8 lines and 80 registers, two
// CTAs an SM, the passes took 38 + 46.
template <class L, int MOST>
struct Share : L {
    static constexpr int T = L::M / L::LEAST;
    static constexpr int LG = MOST >= 3 && T * 8 <= 400 ? 3 : MOST >= 2 && T * 4 <= 400 ? 2 : MOST >= 1 && T * 2 <= 512 ? 1 : 0;
    static constexpr int THREADS = ((T << LG) + 31) / 32 * 32;
    static constexpr int CTAS = 1152 / THREADS > 16 ? 16 : (1152 / THREADS > 1 ? 1152 / THREADS : 1);
    static constexpr int SMEM = (L::M << LG) * (int)sizeof(double2);
};

// One pass of the CTA's lines, radix R, NS = product of the earlier radices.
// ld(k, line) and st(k, line, value) reach global memory.
template <class L, int SIGN, int R, int NS, class LD, class ST>
__device__ __forceinline__ void fft_pass(double2* sm, const double2* tw, const LD& ld, const ST& st) {
    constexpr bool first = NS == 1, last = NS * R == L::M;
    constexpr unsigned nb = L::M / R;
    const unsigned line = threadIdx.x & ((1u << L::LG) - 1), j = threadIdx.x >> L::LG;
    const bool act = j < nb;
    const unsigned k = first ? 0 : j % NS;
    double2 x[R];
    if (act) {
#pragma unroll
        for (unsigned q = 0; q < R; ++q) x[q] = first ? ld(j + q * nb, line) : sm[((j + q * nb) << L::LG) + line];
        if (!first) {
#pragma unroll
            for (unsigned q = 1; q < R; ++q) {
                double2 w = __ldg(tw + q * k * (nb / NS));
                if (SIGN > 0) w.y = -w.y;
                x[q] = c_mul(x[q], w);
            }
        }
        dft<SIGN, R>(x);
    }
    if (!first && !last) __syncthreads();  // every operand is in registers before the buffer is overwritten
    if (act) {
        const unsigned o = (j - k) * R + k;
#pragma unroll
        for (unsigned q = 0; q < R; ++q) {
            if (last) st(o + q * NS, line, x[q]);
            else sm[((o + q * NS) << L::LG) + line] = x[q];
        }
    }
    if (!last) __syncthreads();
}

template <class L, int SIGN, int R0, int R1, int R2, int R3, class LD, class ST>
__device__ __forceinline__ void fft_lines(const Len<R0, R1, R2, R3>&, const double2* tw, const LD& ld, const ST& st) {
    extern __shared__ __align__(16) char fsm[];
    double2* sm = (double2*)fsm;
    fft_pass<L, SIGN, R0, 1>(sm, tw, ld, st);
    fft_pass<L, SIGN, R1, R0>(sm, tw, ld, st);
    fft_pass<L, SIGN, R2, R0 * R1>(sm, tw, ld, st);
    if constexpr (R3 > 1) fft_pass<L, SIGN, R3, R0 * R1 * R2>(sm, tw, ld, st);
}

// Rows along y.  lib = 0: A[f][i][ky] of frame f (real rows of SY pixels).
// lib = 1: the rows of library pair f, p_{2f} - i p_{2f+1}, column v at (v - R/2) mod MY.
template <class L>
__global__ void __launch_bounds__(L::THREADS, L::CTAS) k_fft_rows_fwd(const double2* tw, const double* in, int rows,
                                                                  int cols, int lib, int Z, double2* A) {
    const int i0 = blockIdx.x << L::LG, f = blockIdx.z;
    auto ld = [&](unsigned k, unsigned line) {
        const int i = i0 + line;
        double2 v = make_double2(0, 0);
        if (i < rows) {
            if (!lib) {
                if ((int)k < cols) v.x = in[((size_t)f * rows + i) * cols + k];
            } else {
                const int c = ((int)k + cols / 2) % L::M;
                if (c < cols) {
                    v.x = in[((size_t)(2 * f) * rows + i) * cols + c];
                    if (2 * f + 1 < Z) v.y = -in[((size_t)(2 * f + 1) * rows + i) * cols + c];
                }
            }
        }
        return v;
    };
    auto st = [&](unsigned k, unsigned line, double2 v) {
        if (i0 + (int)line < rows) A[((size_t)f * rows + i0 + line) * L::M + k] = v;
    };
    fft_lines<L, -1>(L(), tw, ld, st);
}

// Columns: row q of A (rows of them, MY wide) sits at (q - shift) mod MX, zeros
// elsewhere; spec[f][kx][ky], conjugated and scaled when conj != 0.
template <class L>
__global__ void __launch_bounds__(L::THREADS, L::CTAS) k_fft_cols_fwd(const double2* tw, const double2* A, int rows,
                                                                  int shift, int MY, double scale, int conj,
                                                                  double2* spec) {
    const int c0 = blockIdx.x << L::LG, f = blockIdx.z;
    auto ld = [&](unsigned k, unsigned line) {
        const int c = c0 + line, q = ((int)k + shift) % L::M;
        return q < rows && c < MY ? A[((size_t)f * rows + q) * MY + c] : make_double2(0, 0);
    };
    auto st = [&](unsigned k, unsigned line, double2 v) {
        if (c0 + (int)line >= MY) return;
        spec[((size_t)f * L::M + k) * MY + c0 + line] =
            conj ? make_double2(v.x * scale, -v.y * scale) : v;
    };
    fft_lines<L, -1>(L(), tw, ld, st);
}

// T[f][pair][i < SX][ky] = inverse column transform of F[f] K[pair].
template <class L>
__global__ void __launch_bounds__(L::THREADS, L::CTAS) k_fft_cols_inv(const double2* tw, const double2* F,
                                                                  const double2* K, int SX, int MY, double2* T) {
    const int c0 = blockIdx.x << L::LG, pr = blockIdx.y, f = blockIdx.z, np = gridDim.y;
    const double2* Ff = F + (size_t)f * L::M * MY;
    const double2* Kp = K + (size_t)pr * L::M * MY;
    double2* To = T + (size_t)(f * np + pr) * SX * MY;
    auto ld = [&](unsigned k, unsigned line) {
        const int c = c0 + line;
        if (c >= MY) return make_double2(0, 0);
        const size_t o = (size_t)k * MY + c;
        return c_mul(Ff[o], Kp[o]);
    };
    auto st = [&](unsigned k, unsigned line, double2 v) {
        if ((int)k < SX && c0 + (int)line < MY) To[(size_t)k * MY + c0 + line] = v;
    };
    fft_lines<L, 1>(L(), tw, ld, st);
}

// Scores of slices 2 pr and 2 pr + 1 from the inverse row transforms of T:
// corr / (sqrt(Mx My) sqrt(varPSF varImage)), -1 / -2 where a variance is not
// positive (as the direct form).  isv: k_det_var.
template <class L>
__global__ void __launch_bounds__(L::THREADS, L::CTAS) k_fft_rows_inv(const double2* tw, const double2* T, DetView V,
                                                                  const double* isv, double* score) {
    const int i0 = blockIdx.x << L::LG, pr = blockIdx.y, f = blockIdx.z, np = gridDim.y;
    const int SX = V.SX, SY = V.SY, r0 = 2 * pr;
    const size_t SS = (size_t)SX * SY;
    const double2* Tp = T + (size_t)(f * np + pr) * SX * L::M;
    const double vp0 = V.varpsf[r0], vp1 = r0 + 1 < V.Z ? V.varpsf[r0 + 1] : 0.0;
    const double a0 = V.inv_m / sqrt(vp0), a1 = V.inv_m / sqrt(vp1);
    double* s0 = score + ((size_t)f * V.Z + r0) * SS;
    auto ld = [&](unsigned k, unsigned line) {
        const int i = i0 + line;
        return i < SX ? Tp[(size_t)i * L::M + k] : make_double2(0, 0);
    };
    auto st = [&](unsigned k, unsigned line, double2 v) {
        const int i = i0 + line;
        if (i >= SX || (int)k >= SY) return;
        const size_t px = (size_t)i * SY + k;
        const double w = isv[f * SS + px];
        s0[px] = w >= 0 && vp0 > 0 ? v.x * a0 * w : (vp0 <= 0 ? -1.0 : -2.0);
        if (r0 + 1 < V.Z) s0[SS + px] = w >= 0 && vp1 > 0 ? v.y * a1 * w : (vp1 <= 0 ? -1.0 : -2.0);
    };
    fft_lines<L, 1>(L(), tw, ld, st);
}

// ------------------------------------------------------------------ host ----

// The line lengths, each at most 12% (above 1024: 33%) over the one before.  Frames
// whose padded side is larger, or smaller than 50 px, take the direct correlation.
#define FFT_LENGTHS(X)                                                                                              \
    X(4, 4, 4, 1) X(5, 4, 4, 1) X(6, 4, 4, 1) X(5, 5, 4, 1) X(6, 5, 4, 1) X(8, 4, 4, 1) X(6, 6, 4, 1) X(6, 5, 5, 1)     \
    X(8, 5, 4, 1) X(6, 6, 5, 1) X(8, 6, 4, 1) X(8, 5, 5, 1) X(6, 6, 6, 1) X(8, 6, 5, 1) X(8, 8, 4, 1) X(8, 6, 6, 1)     \
    X(8, 8, 5, 1) X(8, 8, 6, 1) X(8, 8, 8, 1) X(6, 6, 4, 4) X(8, 5, 4, 4) X(6, 6, 5, 4) X(8, 6, 4, 4) X(6, 6, 6, 4)     \
    X(8, 6, 5, 4) X(8, 8, 4, 4) X(8, 8, 5, 4) X(8, 8, 6, 4) X(8, 8, 8, 4)

static bool fft_length(int n, int* out) {
    int best = 0;
#define X(a, b, c, d)                                                     \
    {                                                                     \
        using L = Len<a, b, c, d>;                                        \
        if (L::M >= n && (best == 0 || L::M < best)) {                    \
            best = L::M;                                                  \
        }                                                                 \
    }
    FFT_LENGTHS(X)
#undef X
    *out = best;
    return best > 0 && n >= 50;
}

// fn(L()) for the length M.
template <class FN>
static void with_len(int M, const FN& fn) {
    switch (M) {
#define X(a, b, c, d) case a * b * c * d: fn(Len<a, b, c, d>()); break;
        FFT_LENGTHS(X)
#undef X
    }
}


// Launch kernel<length M>(...) on grid, grid.x = the lines; kernels are templates, so each
// gets a functor.
#define FFT_LAUNCHER(name, MOST)                                                                                  \
    template <class... ARGS>                                                                                      \
    static void launch_##name(int M, dim3 grid, cudaStream_t st, ARGS... args) {                                  \
        with_len(M, [&](auto len) {                                                                               \
            using L = Share<decltype(len), MOST>;                                                                 \
            grid.x = (grid.x + (1u << L::LG) - 1) >> L::LG;                                                       \
            cudaFuncSetAttribute(k_##name<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);              \
            k_##name<L><<<grid, L::THREADS, L::SMEM, st>>>(args...);                                              \
        });                                                                                                       \
    }
FFT_LAUNCHER(fft_rows_fwd, 1)
FFT_LAUNCHER(fft_cols_fwd, 3)
FFT_LAUNCHER(fft_cols_inv, 3)
FFT_LAUNCHER(fft_rows_inv, 1)

void det_fft_free(DetFft& p) {
    if (p.d_tab) cudaFree(p.d_tab);
    p = DetFft();
}

// Twiddles and library spectra of a detector.  A detector without them (p.d_tab
// null: no memory, or a rule of det_fft_wanted) runs the direct correlation.
void det_fft_build(zola_ctx* ctx, const DetView& v, DetFft& p) {
    p = DetFft();
    if (!det_fft_wanted(v)) return;
    DetFft q;
    if (!fft_length(v.SX + v.R / 2, &q.MX) || !fft_length(v.SY + v.R / 2, &q.MY)) return;
    q.pairs = (v.Z + 1) / 2;
    const size_t MM = (size_t)q.MX * q.MY, nk = MM * q.pairs;
    if (nk * sizeof(double2) > DET_FFT_MAX_LIBRARY) return;
    double2* A = nullptr;
    bool ok = cudaMalloc(&q.d_tab, (q.MX + q.MY + nk) * sizeof(double2)) == cudaSuccess &&
              cudaMalloc(&A, (size_t)q.pairs * v.R * q.MY * sizeof(double2)) == cudaSuccess;
    if (ok) {
        std::vector<double2> tw(q.MX + q.MY);
        for (int k = 0; k < q.MX; ++k) tw[k] = make_double2(std::cos(2 * M_PI * k / q.MX), -std::sin(2 * M_PI * k / q.MX));
        for (int k = 0; k < q.MY; ++k)
            tw[q.MX + k] = make_double2(std::cos(2 * M_PI * k / q.MY), -std::sin(2 * M_PI * k / q.MY));
        ok = cudaMemcpy(q.d_tab, tw.data(), tw.size() * sizeof(double2), cudaMemcpyHostToDevice) == cudaSuccess;
    }
    if (ok) {
        cudaStream_t st = ctx->stream;
        launch_fft_rows_fwd(q.MY, dim3((unsigned)(v.R), 1, q.pairs), st, q.twy(), v.psf0, v.R, v.R, 1, v.Z, A);
        launch_fft_cols_fwd(q.MX, dim3((unsigned)(q.MY), 1, q.pairs), st, q.twx(), A, v.R, v.R / 2, q.MY,
                            1.0 / (double)MM, 1, q.K());
        ctx->launches += 2;
        ok = cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(st) == cudaSuccess;
    }
    if (A) cudaFree(A);
    if (!ok) {
        cudaGetLastError();  // the detector still works without the spectra
        if (q.d_tab) cudaFree(q.d_tab);
        return;
    }
    p = q;
}

// Frames whose T fits in about half of the 126 MB L2 go through the two inverse
// passes together, so that T is read back from L2.
static int frames_together(const DetView& v, const DetFft& p, int nf) {
    const size_t t = (size_t)p.pairs * v.SX * p.MY * sizeof(double2);
    return (int)std::max<size_t>(1, std::min<size_t>((size_t)nf, DET_FFT_T_BYTES / t));
}

size_t det_fft_scratch(const DetView& v, const DetFft& p, int nf) {
    const size_t t = (size_t)p.pairs * v.SX * p.MY * frames_together(v, p, nf), a = (size_t)v.SX * p.MY * nf;
    return (std::max(t, a) + (size_t)p.MX * p.MY * nf) * sizeof(double2);
}

void det_fft_scores(zola_ctx* ctx, const DetView& v, const DetFft& p, const double* frames, int nf, const double* isv,
                    char* scratch, double* score, cudaStream_t st) {
    const int MX = p.MX, MY = p.MY, FS = frames_together(v, p, nf);
    const size_t SS = (size_t)v.SX * v.SY;
    double2* F = (double2*)scratch;                 // spectra of the frames
    double2* T = F + (size_t)MX * MY * nf;          // row transforms, then the inverse column transforms
    launch_fft_rows_fwd(MY, dim3((unsigned)(v.SX), 1, nf), st, p.twy(), frames, v.SX, v.SY, 0, 0, T);
    launch_fft_cols_fwd(MX, dim3((unsigned)(MY), 1, nf), st, p.twx(), T, v.SX, 0, MY, 1.0, 0, F);
    ctx->launches += 2;
    for (int f0 = 0; f0 < nf; f0 += FS) {
        const int n = std::min(FS, nf - f0);
        launch_fft_cols_inv(MX, dim3((unsigned)(MY), p.pairs, n), st, p.twx(), F + (size_t)f0 * MX * MY, p.K(), v.SX,
                            MY, T);
        launch_fft_rows_inv(MY, dim3((unsigned)(v.SX), p.pairs, n), st, p.twy(), T, v, isv + f0 * SS,
                            score + (size_t)f0 * v.Z * SS);
        ctx->launches += 2;
    }
}

}  // namespace zola
