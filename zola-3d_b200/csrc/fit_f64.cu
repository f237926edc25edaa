// Plain FP64 GPU form of the PSF model and of the per-ROI Poisson MLE fit.
//
// One cluster of CTAs per ROI (persistent grid pulling ROIs from a device
// counter), all arithmetic in FP64 on the CUDA cores, no tensor cores.  This is the 1x
// reference the split-precision tcgen05 path is measured against, and the
// FP64 device model that the parity tests compare with the CPU oracle.
//
// The model restates process/cpu/PSFPhase.java:557-629 (pupil -> |IFFT|^2 ->
// circular Gaussian blur -> |.| -> crop -> normalise) as partial DFTs:
//   Q  = pupil * exp(i(kx x + ky y + phase + kz zwat - kzoil zoil))   (D x D)
//   S  = Q C^T,  Sy = Q diag(i ky) C^T,  Sz = (i kz o Q) C^T          (D x W)
//   E  = C S,  Ex = C diag(i kx) S,  Ey = C Sy,  Ez = C Sz            (W x W)
//   I  = |E|^2,  I_t = 2 Re(conj(E) E_t)
//   B  = G I G^T (R x R),  psi = |B| / sum|B|,
//   dpsi_t = (sgn(B) B_t - psi sum sgn(B) B_t) / sum|B|.
// The forward field uses the reference's (cos q, sin r) pair (PSFPhase.java:565-569)
// so evanescent tables built with resetKz are reproduced; derivatives assume
// q == r, which holds for the fit tables (kz = 0 where evanescent).
//
// Two forms of the sums.  FFTs (eval_maps) serve the models and most fits of
// zola_fit_batch.  Where the last bit matters the partial DFTs are summed directly, every
// sum in a fixed order (direct_maps): a fit that meets a flat or singular likelihood (z = 0
// of a PSF that is the same above and below focus, where rounding decides which way it
// turns) amplifies the 1e-15 between the two forms to nanometres, or to the other side of
// focus.  So a fit of zola_fit_batch is taken again, from its start, by direct sums when
// the FFT form does not bring it to convergence in F64_TRIAL evaluations, or meets a point
// where one of x, y, z has less than F64_WEAK of the largest one's Fisher information (z
// within 3 nm of such a focus).  The frame pipeline, whose candidates mostly run long, fits
// by direct sums at once, and its rows take direct models, as do the finite differences
// of CRLB curves.  Of 250,000 fits of six PSFs, from good, poor and z = 0 starts, the others end
// within 1.3e-10 of the direct form's in every parameter and bound, after as many
// evaluations.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "fft_f64.h"
#include "lm.h"
#include "zola_internal.h"

namespace zola {

constexpr int F64_THREADS = FL_THREADS;
constexpr int F64_NRED = 1 + 5 + 15 + 15;  // nll, g, H (lower), F (lower)
constexpr int F64_RED_BYTES = 4096;        // reduction areas at the start of shared memory
constexpr size_t F64_G_SMEM = 56 * 1024;   // blur matrices up to this size are kept in shared memory

// Work areas of a cluster in global memory (they stay in L2).
struct F64Work {
    double2* S;  // 3 * (w, a) planes, W*D
    double* J;   // 4 * R*W
    double* T;   // 4 * R*R: the CTA's rows of map m start at T + m * nt
    int nt;      // pixels of the CTA's rows
};
struct DirectWork {
    double2* Q;  // D*D
    double2* S;  // 3 * D*W
    double* I;   // 4 * W*W
    double* J;   // 4 * R*W
    double* T;   // 4 * R*R
};

__host__ __device__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

__host__ __device__ inline size_t f64_work_bytes(int D, int W, int R) {
    size_t b = 0;
    b += align_up((size_t)3 * D * W * 16, 256);
    b += align_up((size_t)4 * R * W * 8, 256);
    b += align_up((size_t)4 * R * R * 8, 256);
    return b;
}
__host__ __device__ inline size_t direct_work_bytes(int D, int W, int R) {
    return f64_work_bytes(D, W, R) + align_up((size_t)D * D * 16, 256) + align_up((size_t)4 * W * W * 8, 256);
}

__device__ inline F64Work f64_carve(char* base, int D, int W, int R) {
    F64Work w{};
    size_t o = 0;
    w.S = (double2*)(base + o); o += align_up((size_t)3 * D * W * 16, 256);
    w.J = (double*)(base + o);  o += align_up((size_t)4 * R * W * 8, 256);
    w.T = (double*)(base + o);
    return w;
}
__device__ inline DirectWork direct_carve(char* base, int D, int W, int R) {
    const F64Work f = f64_carve(base, D, W, R);
    base += f64_work_bytes(D, W, R);
    return DirectWork{(double2*)base, f.S, (double*)(base + align_up((size_t)D * D * 16, 256)), f.J, f.T};
}

// Shared memory: reduction areas, transform buffer, one tile of the
// pupil field (LINES rows of D | 1) or of an intensity map (W x LINES), and the
// transposed blur matrix (W x R) when it is small enough.
__host__ __device__ inline size_t f64_tile_bytes(int N, int D, int W) {
    const size_t lines = fl_lines(N), q = lines * (D | 1) * 16, x = (size_t)W * lines * 8;
    return align_up(q > x ? q : x, 256);
}
__host__ __device__ inline size_t f64_smem(int N, int D, int W, int R) {
    const size_t g = (size_t)W * R * 8;
    return F64_RED_BYTES + FL_SMEM + f64_tile_bytes(N, D, W) + (g <= F64_G_SMEM ? g : 0);
}


// Pupil field at (row a, column b): pupil (cos q, sin r).
__device__ __forceinline__ double2 pupil_field(const PsfView& P, int a, int b, double x, double y, double zoil, double zwat) {
    const int idx = a * P.D + b;
    const double pup = P.pupil[idx];
    if (pup == 0.0) return make_double2(0.0, 0.0);
    const double pp = P.kx[a] * x + P.ky[b] * y + P.phase[idx];
    const double q = pp + P.kz[idx] * zwat - P.kzoil[idx] * zoil;
    const double r = pp + P.kz[idx] * zwat * P.isim[idx] - P.kzoil[idx] * zoil * P.isimoil[idx];
    double s, c;
    sincos(q, &s, &c);
    if (r != q) s = sin(r);
    return make_double2(pup * c, pup * s);
}

// Computes the four blurred R x R maps T[0..3] = blurred I, I_x, I_y, I_z (only T[0]
// when derivs is false) through N-point FFTs; all threads of the cluster take part.  E[w] = sum_a C[w][a] Q[a] is, up to a
// sign (-1)^(w - W/2) that |E|^2 and conj(E) E_t do not see, output (w - W/2) mod N of
// the inverse N-point transform of Q at points a0 .. a0 + D - 1.  Per LINES pupil rows
// a: Q in shared memory, transforms of Q, i ky Q and i kz Q along b into S (w, a);
// per LINES window columns: transforms of S, i kx S, S_y, S_z along a, E in registers,
// each intensity map straight from registers into a shared tile, blurred along its
// first index there (2 x 2 outputs a thread, two 16-byte loads for four FMAs); then
// the second blur (4 x 2 outputs a thread).
// The direct sums took 8 D W (3 D + 4 W) flops, bound by loads from the work area;
// this takes a sixth of that at N = 128, W = 64 and an eighth at W = 128.  It is bound by
// latency (20% of the FP64 rate with two CTAs an SM: the barriers between passes and the
// reads of S), which is why a cluster shares an evaluation.  200 models with derivatives
// at 32 px (N = 128) 611 -> 124 us; 800 fits of 24 px 15.5 -> 3.8 ms, of which one CTA a
// fit left 6.8; 26 fits of 42 px 8.4 -> 0.75 ms.
template <class F>
__device__ void eval_maps(const Cluster& cl, const PsfView& P, const WinView& Wn, const F64Work& w, char* smem,
                              double x, double y, double zoil, double zwat, bool derivs) {
    constexpr int N = F::N, L = F::LINES;
    const int D = P.D, DP = D | 1, W = Wn.W, R = Wn.R, tid = threadIdx.x, a0 = P.a0;
    double2* buf = (double2*)(smem + F64_RED_BYTES);
    char* tile = smem + F64_RED_BYTES + FL_SMEM;
    double2* Qt = (double2*)tile;  // [row][column]
    double* X = (double*)tile;     // [window row][column]
    const bool gs = (size_t)W * R * 8 <= F64_G_SMEM;
    const double* GT = gs ? (const double*)(tile + f64_tile_bytes(N, D, W)) : Wn.GT;
    const size_t plane = (size_t)W * D;
    // a CTA takes whole tiles of rows, or, where there are fewer tiles than CTAs, fields
    const int nf = derivs ? 3 : 1, tiles = (D + L - 1) / L;
    const bool by_field = tiles < (int)cl.size;
    for (int t = by_field ? 0 : cl.rank; t < tiles; t += by_field ? 1 : cl.size) {
        const int r0 = t * L;
        for (int k = tid; k < L * D; k += FL_THREADS) {
            const int l = k / D, b = k - l * D;
            Qt[l * DP + b] = r0 + l < D ? pupil_field(P, r0 + l, b, x, y, zoil, zwat) : make_double2(0, 0);
        }
        __syncthreads();
        for (int f = by_field ? cl.rank : 0; f < nf; f += by_field ? cl.size : 1) {
            double2* S = w.S + f * plane;
            auto ld = [&](unsigned k, unsigned l) {
                const int b = (int)k - a0;
                if ((unsigned)b >= (unsigned)D) return make_double2(0, 0);
                const double2 q = Qt[l * DP + b];
                if (f == 0) return q;
                const double s = f == 1 ? P.ky[b] : P.kz[min(r0 + (int)l, D - 1) * D + b];
                return make_double2(-s * q.y, s * q.x);
            };
            auto st = [&](unsigned k, unsigned l, int, double2 v) {
                const unsigned o = (k + W / 2) & (N - 1);
                if (o < (unsigned)W && r0 + (int)l < D) S[(size_t)o * D + r0 + l] = v;
            };
            fl_transform<F, 1>(buf, P.tw, ld, st);
            __syncthreads();
        }
        __syncthreads();
    }
    cl.sync();
    for (int c0 = cl.rank * L; c0 < W; c0 += cl.size * L) {
        double2 e[FL_OUT];
        for (int m = 0; m < (derivs ? 4 : 1); ++m) {
            const double2* S = w.S + (m < 2 ? 0 : m - 1) * plane;
            auto ld = [&](unsigned k, unsigned l) {
                const int a = (int)k - a0;
                if ((unsigned)a >= (unsigned)D || c0 + (int)l >= W) return make_double2(0, 0);
                const double2 q = S[(size_t)(c0 + l) * D + a];
                if (m != 1) return q;
                const double s = P.kx[a];
                return make_double2(-s * q.y, s * q.x);
            };
            auto st = [&](unsigned k, unsigned l, int slot, double2 v) {
                const unsigned o = (k + W / 2) & (N - 1);
                if (m == 0) e[slot] = v;
                if (o < (unsigned)W)
                    X[o * L + l] = m == 0 ? v.x * v.x + v.y * v.y : 2.0 * (e[slot].x * v.x + e[slot].y * v.y);
            };
            fl_transform<F, 1>(buf, P.tw, ld, st);
            __syncthreads();
            // J[m][i'][j] = sum_i G[i'][i] I[m][i][j]
            blur_tile(GT, X, R, W, L, min(L, W), w.J + (size_t)m * R * W + c0);
            __syncthreads();
        }
    }
    cl.sync();
    // T[m][i'][j'] = sum_j G[j'][j] J[m][i'][j] for the CTA's rows: two rows i', two maps and two j' a thread
    const int nm = derivs ? 4 : 1, hp = R / 2, i0 = cl.row0(R), pairs = (cl.row1(R) - i0) / 2, mg = derivs ? 2 : 1;
    for (int t = tid; t < pairs * mg * hp; t += FL_THREADS) {
        const int u = t / hp, jp = t - u * hp, ip = u / mg, m0 = 2 * (u - ip * mg), m1 = min(m0 + 1, nm - 1);
        const double* g = GT + 2 * jp;
        const double* j0 = w.J + ((size_t)m0 * R + i0 + 2 * ip) * W;
        const double* j1 = w.J + ((size_t)m1 * R + i0 + 2 * ip) * W;
        double2 s[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = make_double2(0, 0);
#pragma unroll 4
        for (int j = 0; j < W; j += 2) {
            const double2 ga = *(const double2*)(g + (size_t)j * R), gb = *(const double2*)(g + (size_t)(j + 1) * R);
            const double2 v[4] = {*(const double2*)(j0 + j), *(const double2*)(j0 + W + j), *(const double2*)(j1 + j),
                                  *(const double2*)(j1 + W + j)};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s[q].x = fma(gb.x, v[q].y, fma(ga.x, v[q].x, s[q].x));
                s[q].y = fma(gb.y, v[q].y, fma(ga.y, v[q].x, s[q].y));
            }
        }
        double* o = w.T + 2 * ip * R + 2 * jp;
        *(double2*)(o + (size_t)m0 * w.nt) = s[0];
        *(double2*)(o + (size_t)m0 * w.nt + R) = s[1];
        if (m1 != m0) {
            *(double2*)(o + (size_t)m1 * w.nt) = s[2];
            *(double2*)(o + (size_t)m1 * w.nt + R) = s[3];
        }
    }
    __syncthreads();
}

// A CTA's set-up: the work areas of its cluster, T in the transform buffer (free
// when the maps are used) where the CTA's rows fit, and the transposed blur matrix in
// shared memory.
template <int NFFT>
__device__ __forceinline__ F64Work f64_begin(const Cluster& cl, const PsfView& P, const WinView& Wn, char* scratch,
                                             size_t per_cluster, char* smem) {
    F64Work w = f64_carve(scratch + cl.id() * per_cluster, P.D, Wn.W, Wn.R);
    const int i0 = cl.row0(Wn.R);
    w.nt = (cl.row1(Wn.R) - i0) * Wn.R;
    if ((size_t)4 * w.nt * 8 <= FL_SMEM) w.T = (double*)(smem + F64_RED_BYTES);
    else w.T += (size_t)4 * i0 * Wn.R;
    const int n = Wn.W * Wn.R;
    if ((size_t)n * 8 <= F64_G_SMEM) {
        double* g = (double*)(smem + F64_RED_BYTES + FL_SMEM + f64_tile_bytes(NFFT, P.D, Wn.W));
        for (int k = threadIdx.x; k < n; k += FL_THREADS) g[k] = Wn.GT[k];
    }
    __syncthreads();
    return w;
}

// Reduction areas: cluster_sum<36> and cluster_sum<4> have parts of their own.
__device__ inline double* part_lik(double* red) { return red + (FL_WARPS + 1) * F64_NRED; }
__device__ inline double* part_norm(double* red) { return part_lik(red) + F64_NRED; }

// Normalisation sums: S = sum |T0|, Dt = sum sgn(T0) T_t.
__device__ inline void norm_sums(const Cluster& cl, const F64Work& w, bool derivs, double* red, double (&s)[4]) {
    double v[4] = {0, 0, 0, 0};
    const double* T = w.T;
    for (int k = threadIdx.x; k < w.nt; k += blockDim.x) {
        double t0 = T[k];
        double sg = t0 < 0 ? -1.0 : 1.0;
        v[0] += fabs(t0);
        if (derivs) {
            v[1] += sg * T[w.nt + k];
            v[2] += sg * T[2 * w.nt + k];
            v[3] += sg * T[3 * w.nt + k];
        }
    }
    cluster_sum<4>(cl, v, red, part_norm(red));
    for (int k = 0; k < 4; ++k) s[k] = v[k];
}

// Writes psi (and dpsi) of n models; one cluster per model.  With a list, only
// the models list[0 .. *n_dev) are evaluated (position list[m] of xyz, written
// at the same index of out).
template <int NFFT>
__global__ void __launch_bounds__(F64_THREADS, 2) model_f64_kernel(PsfView P, WinView Wn, const double* xyz, int n,
                                                                   double* out, double* dout, char* gscratch,
                                                                   size_t per_cluster, const int* list,
                                                                   const int* n_dev) {
    extern __shared__ __align__(256) char smem_raw[];
    double* red = (double*)smem_raw;
    const Cluster cl;
    const F64Work w = f64_begin<NFFT>(cl, P, Wn, gscratch, per_cluster, smem_raw);
    const int R = Wn.R, nt = w.nt;
    const size_t RR = (size_t)R * R, px0 = (size_t)cl.row0(R) * R;
    const bool derivs = dout != nullptr;
    const int nn = n_dev ? min(n, *n_dev) : n;
    for (int mi = cl.id(); mi < nn; mi += cl.count()) {
        const int m = list ? list[mi] : mi;
        eval_maps<FftLines<NFFT>>(cl, P, Wn, w, smem_raw, xyz[3 * m], xyz[3 * m + 1], P.zfocus, xyz[3 * m + 2], derivs);
        double s[4];
        norm_sums(cl, w, derivs, red, s);
        for (int k = threadIdx.x; k < nt; k += blockDim.x) {
            double t0 = w.T[k];
            double sg = t0 < 0 ? -1.0 : 1.0;
            double psi = fabs(t0) / s[0];
            out[m * RR + px0 + k] = psi;
            if (derivs)
                for (int d = 0; d < 3; ++d)
                    dout[((size_t)m * 3 + d) * RR + px0 + k] = (sg * w.T[(d + 1) * nt + k] - psi * s[d + 1]) / s[0];
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may read its shared memory
}

// ------------------------------------------------------------------------
// The direct form: partial DFT sums in the order of their terms, so that a result never
// depends on how the work is shared.  The threads of a cluster share every pass.
constexpr int DIRECT_THREADS = 512;
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmadd(double2 acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
    return acc;
}

// The four blurred maps as eval_maps, into w.T (map m from m R R on); every thread of the
// cluster.  Bound by the latency of its operands in L2 and by the barriers: 60 us an
// evaluation at N = 128, W = 64 by eight CTAs.  Two outputs a thread: one takes 5.6
// instead of 6.0 ms for 800 fits of 24 px, of which a few go on by direct sums, but twice
// as long where the fits fill the chip; with four it is 7.3 ms.  Tiles of columns kept in
// shared memory by a CTA take 5.4 ms, and a quarter more for a movie.
__device__ void direct_maps(const Cluster& cl, const PsfView& P, const WinView& Wn, const DirectWork& w, double x,
                            double y, double zoil, double zwat, bool derivs) {
    const int D = P.D, W = Wn.W, R = Wn.R, t0 = cl.rank * DIRECT_THREADS + threadIdx.x, nt = cl.size * DIRECT_THREADS;
    for (int idx = t0; idx < D * D; idx += nt) {
        const int a = idx / D, b = idx - a * D;
        const double pup = P.pupil[idx];
        double2 q2 = make_double2(0.0, 0.0);
        if (pup != 0.0) {
            const double pp = P.kx[a] * x + P.ky[b] * y + P.phase[idx];
            const double q = pp + P.kz[idx] * zwat - P.kzoil[idx] * zoil;
            const double r = pp + P.kz[idx] * zwat * P.isim[idx] - P.kzoil[idx] * zoil * P.isimoil[idx];
            q2 = make_double2(pup * cos(q), pup * sin(r));
        }
        w.Q[idx] = q2;
    }
    cl.sync();
    // first contraction over pupil columns b: rows a0 and a0 + 1 of one column j
    constexpr int TA = 2;
    double2 *S = w.S, *Sy = S + (size_t)D * W, *Sz = Sy + (size_t)D * W;
    for (int idx = t0; idx < (D + TA - 1) / TA * W; idx += nt) {
        const int a0 = idx / W * TA, j = idx % W;
        double2 s[TA], sy[TA], sz[TA];
        const double2* q_[TA];
        const double* kz_[TA];
#pragma unroll
        for (int t = 0; t < TA; ++t) {
            s[t] = sy[t] = sz[t] = make_double2(0, 0);
            q_[t] = w.Q + (size_t)min(a0 + t, D - 1) * D;
            kz_[t] = P.kz + (size_t)min(a0 + t, D - 1) * D;
        }
        const double2* crow = Wn.C + (size_t)j * D;
#pragma unroll 4
        for (int b = 0; b < D; ++b) {
            const double2 c = crow[b];
            const double ky = P.ky[b];
#pragma unroll
            for (int t = 0; t < TA; ++t) {
                const double2 qc = cmul(q_[t][b], c);
                s[t].x += qc.x; s[t].y += qc.y;
                if (derivs) {
                    const double kz = kz_[t][b];
                    sy[t].x -= ky * qc.y; sy[t].y += ky * qc.x;   // (i ky) q c
                    sz[t].x -= kz * qc.y; sz[t].y += kz * qc.x;   // (i kz) q c
                }
            }
        }
#pragma unroll
        for (int t = 0; t < TA; ++t) {
            if (a0 + t >= D) break;
            const size_t o = (size_t)(a0 + t) * W + j;
            S[o] = s[t];
            if (derivs) { Sy[o] = sy[t]; Sz[o] = sz[t]; }
        }
    }
    cl.sync();
    // second contraction over pupil rows a, then intensities: rows i0 and i0 + 1 of one column j
    double *I0 = w.I, *I1 = I0 + (size_t)W * W, *I2 = I1 + (size_t)W * W, *I3 = I2 + (size_t)W * W;
    for (int idx = t0; idx < W / TA * W; idx += nt) {
        const int i0 = idx / W * TA, j = idx % W;
        double2 e[TA], ex[TA], ey[TA], ez[TA];
#pragma unroll
        for (int t = 0; t < TA; ++t) e[t] = ex[t] = ey[t] = ez[t] = make_double2(0, 0);
        const double2* c_ = Wn.C + (size_t)i0 * D;
#pragma unroll 4
        for (int a = 0; a < D; ++a) {
            const double2 s = S[(size_t)a * W + j];
            double2 sy = make_double2(0, 0), sz = make_double2(0, 0);
            double kx = 0;
            if (derivs) { sy = Sy[(size_t)a * W + j]; sz = Sz[(size_t)a * W + j]; kx = P.kx[a]; }
#pragma unroll
            for (int t = 0; t < TA; ++t) {
                const double2 c = c_[(size_t)t * D + a];
                const double2 cs = cmul(c, s);
                e[t].x += cs.x; e[t].y += cs.y;
                if (derivs) {
                    ex[t].x -= kx * cs.y; ex[t].y += kx * cs.x;
                    ey[t] = cmadd(ey[t], c, sy);
                    ez[t] = cmadd(ez[t], c, sz);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < TA; ++t) {
            const size_t o = (size_t)(i0 + t) * W + j;
            I0[o] = e[t].x * e[t].x + e[t].y * e[t].y;
            if (derivs) {
                I1[o] = 2.0 * (e[t].x * ex[t].x + e[t].y * ex[t].y);
                I2[o] = 2.0 * (e[t].x * ey[t].x + e[t].y * ey[t].y);
                I3[o] = 2.0 * (e[t].x * ez[t].x + e[t].y * ez[t].y);
            }
        }
    }
    cl.sync();
    // blur along the first index (two rows i' of one column j), then along the second
    const int nm = derivs ? 4 : 1, hp = R / 2;
    for (int idx = t0; idx < nm * hp * W; idx += nt) {
        const int m = idx / (hp * W), rem = idx - m * hp * W, ip = rem / W * 2, j = rem % W;
        const double *Im = w.I + (size_t)m * W * W + j, *g = Wn.G + (size_t)ip * W;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll 8
        for (int i = 0; i < W; ++i) {
            const double v = Im[(size_t)i * W];
            s0 = fma(g[i], v, s0);
            s1 = fma(g[W + i], v, s1);
        }
        w.J[((size_t)m * R + ip) * W + j] = s0;
        w.J[((size_t)m * R + ip + 1) * W + j] = s1;
    }
    cl.sync();
    for (int idx = t0; idx < nm * R * R; idx += nt) {
        const int row = idx / R, jp = idx - row * R;
        const double *g = Wn.GT + jp, *Jm = w.J + (size_t)row * W;
        double s = 0.0;
#pragma unroll 8
        for (int j = 0; j < W; ++j) s = fma(g[(size_t)j * R], Jm[j], s);
        w.T[idx] = s;
    }
    cl.sync();
}

// Sums over n pixels, pixel k to thread k mod 512: pix(k, v) adds a pixel's terms; end(v)
// closes a thread's sums.  Every CTA forms them for itself.  red: 17 NV doubles.
template <int NV, class PIX, class END>
__device__ __forceinline__ void direct_sums(int n, double* red, double (&out)[NV], const PIX& pix, const END& end) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int k = threadIdx.x; k < n; k += DIRECT_THREADS) pix(k, v);
    end(v);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) red[warp * NV + k] = x;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < DIRECT_THREADS / 32; ++w) s += red[w * NV + threadIdx.x];
        red[DIRECT_THREADS / 32 * NV + threadIdx.x] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) out[k] = red[DIRECT_THREADS / 32 * NV + k];
    __syncthreads();
}

__device__ __forceinline__ void direct_norm(const double* T, int RR, bool derivs, double* red, double (&s)[4]) {
    direct_sums<4>(RR, red, s, [&](int k, double (&v)[4]) {
        double t0 = T[k];
        double sg = t0 < 0 ? -1.0 : 1.0;
        v[0] += fabs(t0);
        if (derivs) {
            v[1] += sg * T[RR + k];
            v[2] += sg * T[2 * RR + k];
            v[3] += sg * T[3 * RR + k];
        }
    }, [](double (&)[4]) {});
}

// CTAs a cluster of the direct form for n items: as the window has work for, and fewer
// where the items alone fill the chip.
static int direct_cluster(const zola_ctx* ctx, int W, int n) {
    int c = W >= 64 ? 8 : (W >= 32 ? 4 : 2);
    while (c > 1 && (long long)n * c > ctx->num_sms) c /= 2;
    return c;
}

// The models of model_f64_kernel (without a list) in the direct form.
__global__ void __launch_bounds__(DIRECT_THREADS, 1) model_direct_kernel(PsfView P, WinView Wn, const double* xyz, int n,
                                                                      double* out, double* dout, char* gscratch,
                                                                      size_t per_cluster) {
    __shared__ double red[17 * 4];
    const Cluster cl;
    const DirectWork w = direct_carve(gscratch + cl.id() * per_cluster, P.D, Wn.W, Wn.R);
    const int RR = Wn.R * Wn.R;
    const double* T = w.T;
    const bool derivs = dout != nullptr;
    for (int m = cl.id(); m < n; m += cl.count()) {
        direct_maps(cl, P, Wn, w, xyz[3 * m], xyz[3 * m + 1], P.zfocus, xyz[3 * m + 2], derivs);
        double s[4];
        direct_norm(T, RR, derivs, red, s);
        for (int k = cl.rank * DIRECT_THREADS + threadIdx.x; k < RR; k += cl.size * DIRECT_THREADS) {
            double t0 = T[k];
            double sg = t0 < 0 ? -1.0 : 1.0;
            double psi = fabs(t0) / s[0];
            out[(size_t)m * RR + k] = psi;
            if (derivs)
                for (int d = 0; d < 3; ++d)
                    dout[((size_t)m * 3 + d) * RR + k] = (sg * T[(d + 1) * RR + k] - psi * s[d + 1]) / s[0];
        }
        // (T is written again behind four cluster barriers)
    }
}

// The fits of ROIs list[0 .. *n_dev), or of all n without a list, in the direct form.  FP64
// movies of 13 to 30 frames take 32 (20 frames, 16 px), 88 to 123 (22 to 26 px) and 490 ms
// (38 px); with fits by FFTs, whose rows are not the same, 24, 46 to 58 and 147, and
// with direct sums by one CTA a fit 42, 159 to 194 and 888.
__global__ void __launch_bounds__(DIRECT_THREADS, 1) fit_direct_kernel(PsfView P, WinView Wn, const float* rois,
                                                                    const float* scmos, const double* init, int n,
                                                                    const int* list, const int* n_dev, FitParamsDev prm,
                                                                    double* out5, double* crlb5, double* nll_out,
                                                                    int* st_out, int* it_out, char* gscratch,
                                                                    size_t per_cluster, int* counter, int least,
                                                                    int most) {
    __shared__ double red[17 * F64_NRED];
    __shared__ LMState st;  // every CTA of the cluster steps its own copy, from the same sums
    __shared__ int item, go;
    const Cluster cl;
    const DirectWork w = direct_carve(gscratch + cl.id() * per_cluster, P.D, Wn.W, Wn.R);
    const int RR = Wn.R * Wn.R, items = list ? min(n, *n_dev) : n;
    const double* T = w.T;
    if (items < least || items > most) return;  // (a launch with clusters of another size takes them)
    for (;;) {
        if (cl.rank == 0 && threadIdx.x == 0) item = atomicAdd(counter, 1);
        cl.sync();
        const int i = cl.size > 1 ? cl.read(&item, 0) : item;
        if (i >= items) break;
        const int r = list ? list[i] : i;
        const float* d = rois + (size_t)r * RR;
        const float* sv = scmos ? scmos + (size_t)r * RR : nullptr;
        if (threadIdx.x == 0) {
            for (int q = 0; q < 5; ++q) st.trial[q] = init[5 * (size_t)r + q];
            lm_clamp(st.trial, prm);
            st.status = 0;  // nothing evaluated yet
        }
        __syncthreads();
        do {
            double th[5], s[4], v[F64_NRED];
            for (int q = 0; q < 5; ++q) th[q] = st.trial[q];
            direct_maps(cl, P, Wn, w, th[0], th[1], P.zfocus, th[2], true);
            direct_norm(T, RR, true, red, s);
            const double A = th[3], B = th[4];
            bool bad = false;
            direct_sums<F64_NRED>(RR, red, v, [&](int k, double (&v)[F64_NRED]) {
                double t0 = T[k];
                double sg = t0 < 0 ? -1.0 : 1.0;
                double psi = fabs(t0) / s[0];
                double j[5];
                for (int q = 0; q < 3; ++q) j[q] = A * (sg * T[(q + 1) * RR + k] - psi * s[q + 1]) / s[0];
                j[3] = psi;
                j[4] = 1.0;
                double mu = A * psi + B + (sv ? (double)sv[k] : 0.0);
                if (!(mu > 0.0)) { bad = true; return; }
                double dk = (double)d[k];
                v[0] += dk > 0 ? mu - dk - dk * log(mu / dk) : mu;
                double wg = 1.0 - dk / mu, wh = dk / (mu * mu), wf = 1.0 / mu;
                int o = 1;
#pragma unroll
                for (int q = 0; q < 5; ++q) v[o + q] += wg * j[q];
                o = 6;
#pragma unroll
                for (int q = 0; q < 5; ++q)
#pragma unroll
                    for (int r = 0; r <= q; ++r) {
                        v[o] += wh * j[q] * j[r];
                        v[o + 15] += wf * j[q] * j[r];
                        ++o;
                    }
            }, [&](double (&v)[F64_NRED]) {
                if (bad) v[0] = INFINITY;
                bad = false;
            });
            if (threadIdx.x == 0) {
                double H[25], F[25];
                int o = 6;
                for (int q = 0; q < 5; ++q)
                    for (int r = 0; r <= q; ++r) {
                        H[q * 5 + r] = H[r * 5 + q] = v[o];
                        F[q * 5 + r] = F[r * 5 + q] = v[o + 15];
                        ++o;
                    }
                if (st.status == 0) {
                    for (int q = 0; q < 5; ++q) st.th[q] = th[q];
                    lm_start(st, v[0], v + 1, H, F, prm);
                } else {
                    lm_update(st, v[0], v + 1, H, F, prm);
                }
                go = lm_propose(st, prm) ? 1 : 0;
            }
            __syncthreads();
        } while (go);
        if (cl.rank == 0 && threadIdx.x == 0) {
            for (int q = 0; q < 5; ++q) out5[5 * (size_t)r + q] = st.th[q];
            if (nll_out) nll_out[r] = st.nll;
            if (st_out) st_out[r] = st.status;
            if (it_out) it_out[r] = st.evals;
            if (crlb5) lm_crlb(st.F, crlb5 + 5 * (size_t)r);
        }
        cl.sync();  // item is written again
    }
    cl.sync();  // no CTA leaves while another may read its shared memory
}

// Likelihood, gradient, Gauss-Newton Hessian and Fisher matrix at theta.
// sv (nullable): the ROI's sCMOS term var/gain^2, added to the mean
// (process/cpu/Localization.java:1132).
template <int NFFT>
__device__ void eval_lik_f64(const Cluster& cl, const PsfView& P, const WinView& Wn, const F64Work& w, char* smem,
                             const float* d, const float* sv, const double* th, double* red, double& nll, double* g,
                             double* H, double* F) {
    const int px0 = cl.row0(Wn.R) * Wn.R, nt = w.nt;
    eval_maps<FftLines<NFFT>>(cl, P, Wn, w, smem, th[0], th[1], P.zfocus, th[2], true);
    double s[4];
    norm_sums(cl, w, true, red, s);
    double v[F64_NRED];
#pragma unroll
    for (int k = 0; k < F64_NRED; ++k) v[k] = 0.0;
    const double A = th[3], B = th[4];
    bool bad = false;
    for (int k = threadIdx.x; k < nt; k += blockDim.x) {
        double t0 = w.T[k];
        double sg = t0 < 0 ? -1.0 : 1.0;
        double psi = fabs(t0) / s[0];
        double j[5];
        for (int q = 0; q < 3; ++q) j[q] = A * (sg * w.T[(q + 1) * nt + k] - psi * s[q + 1]) / s[0];
        j[3] = psi;
        j[4] = 1.0;
        double mu = A * psi + B + (sv ? (double)sv[px0 + k] : 0.0);
        if (!(mu > 0.0)) { bad = true; continue; }
        double dk = (double)d[px0 + k];
        v[0] += dk > 0 ? mu - dk - dk * log(mu / dk) : mu;
        double wg = 1.0 - dk / mu, wh = dk / (mu * mu), wf = 1.0 / mu;
        int o = 1;
#pragma unroll
        for (int q = 0; q < 5; ++q) v[o + q] += wg * j[q];
        o = 6;
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
            for (int r = 0; r <= q; ++r) {
                v[o] += wh * j[q] * j[r];
                v[o + 15] += wf * j[q] * j[r];
                ++o;
            }
    }
    if (bad) v[0] = INFINITY;
    cluster_sum<F64_NRED>(cl, v, red, part_lik(red));
    nll = v[0];
    for (int q = 0; q < 5; ++q) g[q] = v[1 + q];
    int o = 6;
    for (int q = 0; q < 5; ++q)
        for (int r = 0; r <= q; ++r) {
            H[q * 5 + r] = H[r * 5 + q] = v[o];
            F[q * 5 + r] = F[r * 5 + q] = v[o + 15];
            ++o;
        }
}

// The trial of every fit; those that go on by direct sums (see above) are listed for
// fit_direct_kernel.  12 evaluations: one to three fits in a hundred go on, and the longer
// the trial, the further the others' rounding travels.  1e-4: with 1e-6 the fits that do
// not go on end up to 7e-11 from the direct form's, with 1e-4 3e-12; 1e-2 takes three times
// as many fits of a saddle-point PSF along.
constexpr int F64_TRIAL = 12;
constexpr double F64_WEAK = 1e-4;
template <int NFFT>
__global__ void __launch_bounds__(F64_THREADS, 2) fit_f64_kernel(PsfView P, WinView Wn, const float* rois,
                                                                 const float* scmos, const double* init, int n,
                                                                 FitParamsDev prm, double* out5, double* crlb5,
                                                                 double* nll_out, int* st_out, int* it_out,
                                                                 char* gscratch, size_t per_cluster, int* counter,
                                                                 int* list, int* listed) {
    extern __shared__ __align__(256) char smem_raw[];
    double* red = (double*)smem_raw;  // reduction area
    __shared__ LMState st;            // every CTA of the cluster steps its own copy, from the same sums
    __shared__ int roi;
    __shared__ int go;
    const Cluster cl;
    const F64Work w = f64_begin<NFFT>(cl, P, Wn, gscratch, per_cluster, smem_raw);
    const int R = Wn.R;
    for (;;) {
        if (cl.rank == 0 && threadIdx.x == 0) roi = atomicAdd(counter, 1);
        cl.sync();
        const int r = cl.size > 1 ? cl.read(&roi, 0) : roi;
        if (r >= n) break;
        const float* d = rois + (size_t)r * R * R;
        const float* sv = scmos ? scmos + (size_t)r * R * R : nullptr;
        if (threadIdx.x == 0) {
            for (int q = 0; q < 5; ++q) st.trial[q] = init[5 * r + q];
            lm_clamp(st.trial, prm);
            st.status = 0;  // nothing evaluated yet
        }
        __syncthreads();
        double th[5], nll, g[5], H[25], F[25];
        do {
            for (int q = 0; q < 5; ++q) th[q] = st.trial[q];
            eval_lik_f64<NFFT>(cl, P, Wn, w, smem_raw, d, sv, th, red, nll, g, H, F);
            if (threadIdx.x == 0) {
                if (st.status == 0) {
                    for (int q = 0; q < 5; ++q) st.th[q] = th[q];
                    lm_start(st, nll, g, H, F, prm);
                } else {
                    lm_update(st, nll, g, H, F, prm);
                }
                go = lm_propose(st, prm) ? 1 : 0;
                if (fmin(F[0], fmin(F[6], F[12])) < F64_WEAK * fmax(F[0], fmax(F[6], F[12]))) {
                    st.status = ZOLA_FIT_MAXITER;
                    go = 0;
                }
            }
            __syncthreads();
        } while (go);
        if (cl.rank == 0 && threadIdx.x == 0) {
            if (st.status != ZOLA_FIT_CONVERGED) {
                list[atomicAdd(listed, 1)] = r;
            } else {
                for (int q = 0; q < 5; ++q) out5[5 * r + q] = st.th[q];
                if (nll_out) nll_out[r] = st.nll;
                if (st_out) st_out[r] = st.status;
                if (it_out) it_out[r] = st.evals;
                if (crlb5) lm_crlb(st.F, crlb5 + 5 * r);
            }
        }
        cl.sync();  // roi is written again
    }
    cl.sync();  // no CTA leaves while another may read its shared memory
}

// Device memory for a launch on st.  Windows whose direct form takes 192 KB have it from
// the context's pool, in the order of the stream, so that their models and fits may run on
// several streams at once, beside other users of the scratch, and be captured at any time
// (they once had no memory but a CTA's shared one).  Larger windows share the scratch.
struct F64Area {
    zola_ctx* ctx;
    cudaStream_t st;
    bool own;
    void* p = nullptr;
    bool failed = false;
    F64Area(zola_ctx* c, const zola_psf* psf, const WindowTables* w, cudaStream_t s)
        : ctx(c), st(s), own(direct_work_bytes(psf->D, w->W, w->R) <= 192 * 1024) {}
    F64Area(const F64Area&) = delete;
    F64Area& operator=(const F64Area&) = delete;
    ~F64Area() { if (p) cudaFreeAsync(p, st); }
    char* get(size_t bytes) {
        if (!own) {
            failed = ensure_scratch(ctx, bytes, ctx->err) != 0;
            return failed ? nullptr : (char*)ctx->scratch;
        }
        const cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, ctx->pool, st);
        if (e == cudaSuccess) return (char*)p;
        failed = true;
        p = nullptr;
        ctx->err = std::string("work area: ") + cudaGetErrorString(e);
        cudaGetLastError();
        return nullptr;
    }
};

// Launch configuration for n ROIs or models in clusters of C CTAs: as many clusters as run
// at once (at most `most`).  attr and cfg live as long as the launch.
template <class K>
static cudaError_t f64_config(K kernel, int C, int threads, size_t smem, int n, long long most, cudaStream_t st,
                              cudaLaunchAttribute* attr, cudaLaunchConfig_t* cfg, int* clusters) {
    *cfg = cudaLaunchConfig_t();
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = C;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
    cfg->blockDim = dim3(threads);
    cfg->gridDim = dim3(C);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int at_once = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&at_once, kernel, cfg);
    *clusters = (int)std::min<long long>(std::min(n, std::max(1, at_once)), most);
    cfg->gridDim = dim3(C * *clusters);
    return e;
}

int launch_model_f64(zola_ctx* ctx, zola_psf* p, WindowTables* w, const double* d_xyz, int n, double* d_out,
                     double* d_dout, cudaStream_t st, const int* d_list, const int* d_count) {
    if (n <= 0) return ZOLA_OK;
    const size_t per_cluster = f64_work_bytes(p->D, w->W, w->R);
    WinView wv{w->R, w->W, w->d_C, w->d_G, w->d_GT};
    int rc = ZOLA_OK;
    F64Area area(ctx, p, w, st);
    with_fft(p->N, [&](auto nfft) {
        auto kernel = model_f64_kernel<decltype(nfft)::value>;
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg;
        int clusters = 0;
        cudaError_t e = f64_config(kernel, f64_cluster(p->N, w->W), F64_THREADS, f64_smem(p->N, p->D, w->W, w->R), n, n, st, &attr,
                                   &cfg, &clusters);
        char* work = e == cudaSuccess ? area.get(per_cluster * (size_t)clusters) : nullptr;
        if (area.failed) { rc = ZOLA_E_CUDA; return; }
        prof_begin(ctx, 6, st);
        if (e == cudaSuccess)
            e = cudaLaunchKernelEx(&cfg, kernel, p->view, wv, d_xyz, n, d_out, d_dout, work, per_cluster, d_list, d_count);
        prof_end(ctx, st);
        if (e != cudaSuccess) { ctx->err = std::string("model: ") + cudaGetErrorString(e); rc = ZOLA_E_CUDA; }
    });
    if (rc) return rc;
    ctx->launches++;
    ZOLA_CUDA_CHECK(cudaGetLastError(), ctx);
    return ZOLA_OK;
}

int launch_model_direct(zola_ctx* ctx, zola_psf* p, WindowTables* w, const double* d_xyz, int n, double* d_out,
                        double* d_dout, cudaStream_t st) {
    if (n <= 0) return ZOLA_OK;
    const size_t per_cluster = direct_work_bytes(p->D, w->W, w->R);
    WinView wv{w->R, w->W, w->d_C, w->d_G, w->d_GT};
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg;
    int clusters = 0;
    cudaError_t e = f64_config(model_direct_kernel, direct_cluster(ctx, w->W, n), DIRECT_THREADS, 0, n, n, st, &attr, &cfg, &clusters);
    if (e == cudaSuccess && ensure_scratch(ctx, per_cluster * (size_t)clusters, ctx->err)) return ZOLA_E_CUDA;
    prof_begin(ctx, 6, st);
    if (e == cudaSuccess)
        e = cudaLaunchKernelEx(&cfg, model_direct_kernel, p->view, wv, d_xyz, n, d_out, d_dout, (char*)ctx->scratch,
                               per_cluster);
    prof_end(ctx, st);
    if (e != cudaSuccess) { ctx->err = std::string("model: ") + cudaGetErrorString(e); return ZOLA_E_CUDA; }
    ctx->launches++;
    return ZOLA_OK;
}

// The kernels of an FP64 fit with their work in area(bytes): counters, the list of fits that
// go on by direct sums, and the clusters' work areas.  room (0: whatever is asked for) bounds
// it: fewer clusters and a shorter list then, and the ROIs in as many pieces as the list
// needs.  direct: no trial by FFTs.
struct F64Fit {
    const float *rois, *scmos;
    const double* init;
    int n;
    double *out5, *crlb5, *nll;
    int *status, *iters;
};
template <class AREA>
static cudaError_t fit_f64_launch(zola_ctx* ctx, const zola_psf* p, const WindowTables* w, const F64Fit& F,
                                  FitParamsDev fp, bool direct, size_t room, cudaStream_t st, const AREA& area) {
    const size_t per_fft = f64_work_bytes(p->D, w->W, w->R), per_direct = direct_work_bytes(p->D, w->W, w->R);
    constexpr size_t HEAD = 256;
    constexpr int PIECE = 1 << 20;
    const WinView wv{w->R, w->W, w->d_C, w->d_G, w->d_GT};
    cudaError_t e = cudaSuccess;
    int piece = direct ? F.n : std::min(F.n, PIECE);
    if (!direct && room) {  // what one work area leaves; too little for a list: direct sums
        const size_t left = (room - HEAD - per_direct) / 256 * 256 / sizeof(int);
        if (left < 4096) direct = true;
        else piece = (int)std::min<size_t>(piece, left);
        if (direct) piece = F.n;
    }
    const size_t list_b = direct ? 0 : align_up((size_t)piece * sizeof(int), 256);
    const size_t most = room ? room - HEAD - list_b : 0;
    // The direct form: with n known, the clusters that suit it; for a list, a launch each with
    // large, small and single-CTA clusters, of which the list's length picks one (3,000 fits of
    // 16 px that all go on: 90 ms by clusters of four, 21 by single CTAs).
    struct { int ctas, least, most, clusters; cudaLaunchAttribute attr; cudaLaunchConfig_t cfg; } D[3];
    int nd = 0, cd = 0;
    if (direct) {
        D[nd++] = {direct_cluster(ctx, w->W, piece), 0, piece};
    } else {
        const int big = direct_cluster(ctx, w->W, 1), to[3] = {ctx->num_sms / 4, ctx->num_sms, piece};
        for (int c = big, k = 0, from = 1; k < 3; from = to[k] + 1, ++k) {
            D[nd++] = {c, from, to[k]};
            c = k == 0 ? std::min(c, 2) : 1;
        }
    }
    cudaLaunchAttribute attr_f;
    cudaLaunchConfig_t cfg_f;
    int cf = 0;
    for (int k = 0; k < nd && e == cudaSuccess; ++k) {
        e = f64_config(fit_direct_kernel, D[k].ctas, DIRECT_THREADS, 0, std::min(piece, D[k].most),
                       room ? most / per_direct : piece, st, &D[k].attr, &D[k].cfg, &D[k].clusters);
        cd = std::max(cd, D[k].clusters);
    }
    if (e != cudaSuccess) return e;
    with_fft(p->N, [&](auto nfft) {
        auto kernel = fit_f64_kernel<decltype(nfft)::value>;
        if (!direct)
            e = f64_config(kernel, f64_cluster(p->N, w->W), F64_THREADS, f64_smem(p->N, p->D, w->W, w->R), piece,
                           room ? most / per_fft : piece, st, &attr_f, &cfg_f, &cf);
        char* base = e == cudaSuccess ? area(HEAD + list_b + std::max(cf * per_fft, cd * per_direct)) : nullptr;
        if (!base) return;
        int *counters = (int*)base, *list = (int*)(base + HEAD);  // FFT queue, list, direct queue
        char* work = base + HEAD + list_b;
        FitParamsDev trial = fp;
        trial.max_iter = std::min(fp.max_iter, F64_TRIAL);
        const size_t RR = (size_t)w->R * w->R;
        for (int a = 0; a < F.n && e == cudaSuccess; a += piece) {
            const int n = std::min(piece, F.n - a);
            const float *rois = F.rois + a * RR, *scmos = F.scmos ? F.scmos + a * RR : nullptr;
            const double* init = F.init + 5 * (size_t)a;
            double *out5 = F.out5 + 5 * (size_t)a, *crlb5 = F.crlb5 ? F.crlb5 + 5 * (size_t)a : nullptr,
                   *nll = F.nll ? F.nll + a : nullptr;
            int *status = F.status ? F.status + a : nullptr, *iters = F.iters ? F.iters + a : nullptr;
            e = cudaMemsetAsync(counters, 0, 3 * sizeof(int), st);
            if (!direct && e == cudaSuccess) {
                e = cudaLaunchKernelEx(&cfg_f, kernel, p->view, wv, rois, scmos, init, n, trial, out5, crlb5, nll, status,
                                       iters, work, per_fft, counters, list, counters + 1);
                ctx->launches++;
            }
            for (int k = 0; k < nd && e == cudaSuccess; ++k) {
                e = cudaLaunchKernelEx(&D[k].cfg, fit_direct_kernel, p->view, wv, rois, scmos, init, n,
                                       direct ? (const int*)nullptr : (const int*)list, (const int*)(counters + 1), fp,
                                       out5, crlb5, nll, status, iters, work, per_direct, counters + 2, D[k].least,
                                       D[k].most);
                ctx->launches++;
            }
        }
    });
    return e;
}

int launch_fit_f64(zola_ctx* ctx, zola_psf* p, WindowTables* w, const float* d_rois, const float* d_scmos,
                   const double* d_init, int n, const zola_fit_params* prm, double* d_out5, double* d_crlb5,
                   double* d_nll, int* d_status, int* d_iters, cudaStream_t st, bool direct) {
    if (n <= 0) return ZOLA_OK;
    FitParamsDev fp{prm->zmin, prm->zmax, prm->xymax, prm->tol_xyz, prm->step_xy, prm->step_z, prm->max_iter};
    const F64Fit F{d_rois, d_scmos, d_init, n, d_out5, d_crlb5, d_nll, d_status, d_iters};
    F64Area area(ctx, p, w, st);
    prof_begin(ctx, 5, st);
    const cudaError_t e =
        fit_f64_launch(ctx, p, w, F, fp, direct, 0, st, [&](size_t bytes) { return area.get(bytes); });
    prof_end(ctx, st);
    if (area.failed) return ZOLA_E_CUDA;
    if (e != cudaSuccess) { ctx->err = std::string("fit: ") + cudaGetErrorString(e); return ZOLA_E_CUDA; }
    ZOLA_CUDA_CHECK(cudaGetLastError(), ctx);
    return ZOLA_OK;
}

}  // namespace zola

// ------------------------------------------------------------------------
// Allocation-free FP64 fit.
//
// Some callers cannot allocate device memory at the time they fit: a host
// application that reserves all device memory for itself at start-up and hands
// plugins only the buffers it owns, or an acquisition thread that must not
// stall on cudaMalloc / cudaFree (both can synchronise the whole device).  For
// them zola_fit_batch_noalloc runs the plain FP64 fit with its per-block work
// areas and its ROI-queue counter in the file-scope array below instead of the
// context's scratch.  The array is part of the library image: every GPU on
// which the library is loaded holds its NOALLOC_SCRATCH_BYTES until the
// process exits.  All calls share it, and it keeps the previous call's
// contents (the counter is cleared at the start of every call), so calls whose
// work overlaps on the GPU (other streams, other host threads) race; serialise
// them.
namespace zola {
constexpr size_t NOALLOC_SCRATCH_BYTES = (size_t)64 << 20;  // 64 MiB
}  // namespace zola

static __device__ __align__(256) unsigned char g_fit_noalloc_scratch[zola::NOALLOC_SCRATCH_BYTES];

namespace {
std::mutex g_noalloc_mu;
// One cached device address per (device, CUDA context): a context that was
// destroyed and created again (cudaDeviceReset, or the primary context
// released and retained again) gets its address looked up afresh.
struct NoallocEntry {
    void* context = nullptr;
    void* ptr = nullptr;
};
NoallocEntry g_noalloc[64];

// The current CUDA context of the calling thread, through the driver entry
// point the runtime exposes (no link against the driver library).
void* current_context() {
    typedef int (*CtxGetCurrent)(void**);
    static CtxGetCurrent fn = nullptr;
    static bool looked = false;
    if (!looked) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (CtxGetCurrent)f;
        looked = true;
    }
    void* c = nullptr;
    if (fn && fn(&c) != 0) c = nullptr;
    return c;
}

// Every kernel that a call may need, of every pupil grid, launched once on no ROIs: a
// kernel's first launch loads it, and may enlarge the stacks, which takes device memory (2 MB
// for one grid of seven).  base: the array.
cudaError_t noalloc_load(const zola_psf& p, const zola::WindowTables& w, char* base, cudaStream_t st) {
    using namespace zola;
    PsfView P = p.view;
    P.D = 4;
    const WinView wv{4, 4, w.d_C, w.d_G, w.d_GT};  // (its tables are at least as large)
    const FitParamsDev fp{};
    int* counter = (int*)base;
    cudaError_t e = cudaMemsetAsync(counter, 0, 3 * sizeof(int), st);
    for (int N = 4; N <= 1024 && e == cudaSuccess; N *= 2)
        with_fft(N, [&](auto nfft) {
            auto kernel = fit_f64_kernel<decltype(nfft)::value>;
            const size_t smem = f64_smem(N, P.D, wv.W, wv.R);
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return;
            kernel<<<1, F64_THREADS, smem, st>>>(P, wv, nullptr, nullptr, nullptr, 0, fp, nullptr, nullptr, nullptr, nullptr,
                                                 nullptr, base + 256, 0, counter, nullptr, nullptr);
            e = cudaGetLastError();
        });
    if (e != cudaSuccess) return e;
    fit_direct_kernel<<<1, DIRECT_THREADS, 0, st>>>(P, wv, nullptr, nullptr, nullptr, 0, nullptr, nullptr, fp, nullptr,
                                                    nullptr, nullptr, nullptr, nullptr, base + 256, 0, counter + 2, 0, 0);
    return cudaGetLastError();
}

// Device address of the scratch array in the current context (host code must
// not use the array's name as a device pointer).  Looked up once per device
// and context, when *fresh is set; the caller has made the device current.
void* noalloc_scratch(int device, std::string& err, bool* fresh) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (device < 0 || device >= 64) {
        err = "zola_fit_batch_noalloc: device index out of range";
        return nullptr;
    }
    void* c = current_context();
    NoallocEntry& e = g_noalloc[device];
    *fresh = !e.ptr || c != e.context;
    if (*fresh) {
        void* p = nullptr;
        cudaError_t rc = cudaGetSymbolAddress(&p, g_fit_noalloc_scratch);
        if (rc != cudaSuccess || !p) {
            err = std::string("zola_fit_batch_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(rc);
            return nullptr;
        }
        e.ptr = p;
        e.context = c;
    }
    return e.ptr;
}
}  // namespace

extern "C" int zola_fit_batch_noalloc(zola_psf* psf, int R, const float* d_rois, const double* d_init5, int n,
                                      const zola_fit_params* prm, double* d_out5, double* d_crlb5, double* d_nll,
                                      int* d_status, int* d_iters, void* stream) {
    using namespace zola;
    if (!psf) return ZOLA_E_ARG;
    zola_ctx* ctx = psf->ctx;
    if (!prm || prm->precision != ZOLA_PREC_FP64 || prm->max_iter < 1 || prm->max_iter > 1000 ||
        !(prm->zmax >= prm->zmin) || !(prm->xymax > 0) || !(prm->step_xy > 0) || !(prm->step_z > 0) ||
        !(prm->tol_xyz >= 0)) {
        ctx->err = "zola_fit_batch_noalloc: needs valid FP64 fit params (precision = ZOLA_PREC_FP64)";
        return ZOLA_E_ARG;
    }
    if (n < 0 || (n > 0 && (!d_rois || !d_init5 || !d_out5))) {
        ctx->err = "zola_fit_batch_noalloc: bad n or null buffer";
        return ZOLA_E_ARG;
    }
    if (psf->o.kz_reset) {
        ctx->err = "zola_fit_batch_noalloc: fit needs a PSF built with kz_reset = 0";
        return ZOLA_E_ARG;
    }
    // Only look the window tables up: building them would allocate.
    auto it = psf->win.find(R);
    if (it == psf->win.end()) {
        ctx->err = "zola_fit_batch_noalloc: tables for this ROI size are not prepared; call "
                   "zola_psf_model_dev(psf, R, NULL, 0, NULL, NULL, stream) once beforehand";
        return ZOLA_E_ARG;
    }
    WindowTables* w = &it->second;
    if (n == 0) return ZOLA_OK;
    // the PSF's device, as every other entry point (no allocation once its context exists)
    if (cudaSetDevice(ctx->device) != cudaSuccess) {
        ctx->err = "zola_fit_batch_noalloc: cudaSetDevice failed";
        return ZOLA_E_CUDA;
    }
    bool fresh = false;
    char* base = (char*)noalloc_scratch(ctx->device, ctx->err, &fresh);
    if (!base) return ZOLA_E_CUDA;
    const size_t per_cluster = direct_work_bytes(psf->D, w->W, w->R);
    if (per_cluster > NOALLOC_SCRATCH_BYTES - 256) {
        ctx->err = "zola_fit_batch_noalloc: one block's work area (" + std::to_string(per_cluster) +
                   " bytes for this ROI size) exceeds the 64 MiB static scratch";
        return ZOLA_E_ARG;
    }
    cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
    FitParamsDev fp{prm->zmin, prm->zmax, prm->xymax, prm->tol_xyz, prm->step_xy, prm->step_z, prm->max_iter};
    const F64Fit F{d_rois, nullptr, d_init5, n, d_out5, d_crlb5, d_nll, d_status, d_iters};
    cudaError_t e = fresh ? noalloc_load(*psf, *w, base, st) : cudaSuccess;
    if (e == cudaSuccess)
        e = fit_f64_launch(ctx, psf, w, F, fp, false, NOALLOC_SCRATCH_BYTES, st, [&](size_t) { return base; });
    if (e != cudaSuccess) {
        ctx->err = std::string("zola_fit_batch_noalloc: ") + cudaGetErrorString(e);
        return ZOLA_E_CUDA;
    }
    return ZOLA_OK;
}
