// Library PSFs of a detector: the FP64 model at x = y = 0 over a range of depths, as
// direct partial DFTs with every sum in a fixed order, made once per detector.
//
// The starts of the pipeline's fits are refined against these images, and a split fit's
// path depends on the last bit of its start: with a library from the FFT form of the same
// model (fit_f64.cu), 1e-15 away, four of a hundred localizations of 40 px ended up to
// 10 nm elsewhere on the flat floor of their likelihood.  So this form stays as it is, and
// a movie's fits start from the same bits whatever form the model takes.  (Its FP64 fits
// are as sensitive by themselves; fit_f64.cu takes them by direct sums too.)
#include <cuda_runtime.h>

#include <algorithm>

#include "zola_internal.h"

namespace zola {

constexpr int LIB_THREADS = 512, LIB_WARPS = LIB_THREADS / 32;

// A CTA's work area: pupil field (D x D), first contraction (D x W), intensity (W x W),
// and the blur's two passes (R x W, R x R).
static __host__ __device__ size_t lib_work(int D, int W, int R) {
    return (size_t)2 * D * D + (size_t)2 * D * W + (size_t)W * W + (size_t)R * W + (size_t)R * R;
}

__device__ inline double2 lib_cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__global__ void __launch_bounds__(LIB_THREADS) k_library(PsfView P, WinView Wn, const double* zwats, int n, double* out,
                                                         double* work) {
    const int D = P.D, W = Wn.W, R = Wn.R, tid = threadIdx.x, nt = LIB_THREADS;
    __shared__ double red[LIB_WARPS];
    double2* Q = (double2*)(work + blockIdx.x * lib_work(D, W, R));
    double2* S = Q + (size_t)D * D;
    double* I = (double*)(S + (size_t)D * W);
    double* J = I + (size_t)W * W;
    double* T = J + (size_t)R * W;
    const double x = 0.0, y = 0.0, zoil = P.zfocus;
    for (int m = blockIdx.x; m < n; m += gridDim.x) {
        const double zwat = zwats[m];
        for (int idx = tid; idx < D * D; idx += nt) {
            const int a = idx / D, b = idx - a * D;
            const double pup = P.pupil[idx];
            double2 q2 = make_double2(0.0, 0.0);
            if (pup != 0.0) {
                const double pp = P.kx[a] * x + P.ky[b] * y + P.phase[idx];
                const double q = pp + P.kz[idx] * zwat - P.kzoil[idx] * zoil;
                const double r = pp + P.kz[idx] * zwat * P.isim[idx] - P.kzoil[idx] * zoil * P.isimoil[idx];
                q2 = make_double2(pup * cos(q), pup * sin(r));
            }
            Q[idx] = q2;
        }
        __syncthreads();
        // S = Q C^T, then E = C S and |E|^2: four rows of a column a thread, terms in order
        constexpr int TA = 4;
        for (int idx = tid; idx < (D + TA - 1) / TA * W; idx += nt) {
            const int a0 = idx / W * TA, j = idx % W;
            double2 s[TA];
#pragma unroll
            for (int t = 0; t < TA; ++t) s[t] = make_double2(0, 0);
            for (int b = 0; b < D; ++b) {
                const double2 c = Wn.C[(size_t)j * D + b];
#pragma unroll
                for (int t = 0; t < TA; ++t) {
                    if (a0 + t >= D) break;
                    const double2 qc = lib_cmul(Q[(size_t)(a0 + t) * D + b], c);
                    s[t].x += qc.x;
                    s[t].y += qc.y;
                }
            }
#pragma unroll
            for (int t = 0; t < TA; ++t)
                if (a0 + t < D) S[(size_t)(a0 + t) * W + j] = s[t];
        }
        __syncthreads();
        for (int idx = tid; idx < W / TA * W; idx += nt) {
            const int i0 = idx / W * TA, j = idx % W;
            double2 e[TA];
#pragma unroll
            for (int t = 0; t < TA; ++t) e[t] = make_double2(0, 0);
            for (int a = 0; a < D; ++a) {
                const double2 s = S[(size_t)a * W + j];
#pragma unroll
                for (int t = 0; t < TA; ++t) {
                    const double2 cs = lib_cmul(Wn.C[(size_t)(i0 + t) * D + a], s);
                    e[t].x += cs.x;
                    e[t].y += cs.y;
                }
            }
#pragma unroll
            for (int t = 0; t < TA; ++t) I[(size_t)(i0 + t) * W + j] = e[t].x * e[t].x + e[t].y * e[t].y;
        }
        __syncthreads();
        // blur along the first index, then along the second
        for (int idx = tid; idx < R * W; idx += nt) {
            const int ip = idx / W, j = idx % W;
            double acc = 0.0;
            for (int i = 0; i < W; ++i) acc = fma(Wn.G[(size_t)ip * W + i], I[(size_t)i * W + j], acc);
            J[idx] = acc;
        }
        __syncthreads();
        for (int idx = tid; idx < R * R; idx += nt) {
            const int ip = idx / R, jp = idx % R;
            double acc = 0.0;
            for (int j = 0; j < W; ++j) acc = fma(Wn.G[(size_t)jp * W + j], J[(size_t)ip * W + j], acc);
            T[idx] = acc;
        }
        __syncthreads();
        double v = 0.0;
        for (int k = tid; k < R * R; k += nt) v += fabs(T[k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) red[tid >> 5] = v;
        __syncthreads();
        double sum = 0.0;
        for (int w = 0; w < LIB_WARPS; ++w) sum += red[w];
        for (int k = tid; k < R * R; k += nt) out[(size_t)m * R * R + k] = fabs(T[k]) / sum;
        __syncthreads();  // the work area is written again
    }
}

int library_psfs(zola_psf* psf, int R, const double* zwat, int n, double* out) {
    zola_ctx* ctx = psf->ctx;
    if (R < 4 || R % 2 || R > psf->N) {
        ctx->err = "ROI side must be even, >= 4 and <= the pupil grid";
        return ZOLA_E_ARG;
    }
    cudaSetDevice(ctx->device);
    WindowTables* w = get_window(psf, R, ctx->err);
    if (!w) return ZOLA_E_ARG;
    const size_t rr = (size_t)R * R, area = lib_work(psf->D, w->W, R);
    const int blocks = std::min(n, 2 * ctx->num_sms);
    double* d = nullptr;  // depths, images, work areas
    const size_t nz = ((size_t)n + 1) / 2 * 2;  // (R and W are even: the areas' complex values are aligned)
    ZOLA_CUDA_CHECK(cudaMalloc(&d, (nz + rr * n + area * blocks) * sizeof(double)), ctx);
    cudaError_t e = cudaMemcpyAsync(d, zwat, (size_t)n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        WinView wv{w->R, w->W, w->d_C, w->d_G, w->d_GT};
        k_library<<<blocks, LIB_THREADS, 0, ctx->stream>>>(psf->view, wv, d, n, d + nz, d + nz + rr * n);
        ctx->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out, d + nz, rr * n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    cudaFree(d);
    ZOLA_CUDA_CHECK(e, ctx);
    return ZOLA_OK;
}

}  // namespace zola
