// Zernike PSF calibration from bead z-stacks: FP64 forward model, hand-written
// adjoint (reverse mode), forward-mode tangents, a Gauss-Newton matrix built on
// the device, and an FP64 Levenberg-Marquardt driver.
//
// Model (process/cpu/ZernikePhaseRetrieval.java:1843-1874, background
// :1519-1530): for bead b and slice s, the PSF psi at (x_b, y_b,
// zoil = dz_s + z_b, zwat = 0) with phase sum_i a_i Z_i over modes i >= 3
// (modes 0-2 are the per-bead registration, :93-95, carried here as x_b, y_b,
// z_b) and blur width sigma;
//   mu = psi (A0_bs + a_bs) + sum_k c_bk m_k(i, ii),  m = 1, i, i^2, ii, i ii, ii^2
// (A0 from InitBackgroundAndPhotonNumber, the reference's fit_a + fit_a_each
// folded into a_bs, PolynomialBackground of order 2); mu <= 0 is replaced by
// 1e-8 (:1862-1864) and contributes no gradient; NLL = sum mu - d ln mu.
// The reference updates one parameter at a time by finite-difference Newton
// steps (:225-300, 860-1050, 1081-1198).  Here the gradient of the whole stack
// NLL comes from one adjoint pass per slice:
//   w = 1 - d/mu;  g_psi = At w;  g_m = (g_psi - sum g_psi psi) / S;  g_T = sgn(T) g_m
//   dNLL/dsigma = <g_T, dG I G^T + G I dG^T>
//   g_I = G^T g_T G;  Ebar = g_I o E;  Qbar = C^H Ebar conj(C)
//   g_phi = 2 Im(conj(Q) Qbar)   (per pupil pixel)
//   dNLL/da_i = sum g_phi Z_i,  dNLL/dx_b = sum g_phi kx,  dNLL/dy_b = sum g_phi ky,
//   dNLL/dz_b = -sum g_phi kzoil,  dNLL/da_bs = sum w psi,  dNLL/dc_bk = sum w m_k.
// Tangents (for the Gauss-Newton matrix) push a phase direction dphi through
// dQ = i Q dphi, dE = C dQ C^T, dI = 2 Re(conj E dE), dT = G dI G^T (or
// dT = dG I G^T + G I dG^T for sigma), dpsi = (sgn T dT - psi sum sgn T dT) / S.
// C and C^H are N-point transforms (fft_f64.h): up to signs (-1)^(i - W/2) (-1)^(j - W/2)
// on E, which |E|^2, conj(E) dE and C^H (g_I o E) conj(C) do not see, E(i, j) is output
// (i - W/2, j - W/2) mod N of the inverse transform of Q at points a0 .. a0 + D - 1.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fft_f64.h"
#include "zola_internal.h"

namespace zola {

constexpr int NPOLY = 6;
constexpr int NOUT = 6 + NPOLY;  // per slice: nll, d/da_bs, d/dsigma, d/dc_k, d/dx, d/dy, d/dz

__host__ __device__ inline double poly_m(int k, int i, int ii) {
    switch (k) {
        case 0: return 1.0;
        case 1: return (double)i;
        case 2: return (double)i * i;
        case 3: return (double)ii;
        case 4: return (double)i * ii;
        default: return (double)ii * ii;
    }
}

struct CalView {
    int D, a0, W, R, nb, ns, pb;  // pb = per-bead stride 3 + ns + NPOLY
    const double* pupil;          // D x D
    const double* kx;             // D
    const double* ky;             // D
    const double* kzoil;          // D x D
    const double2* tw;            // N
    const double* GT;             // W x R: blur matrix at the current sigma, transposed
    const double* dGT;            // W x R: its derivative by sigma
    const double* dz;             // ns
    const double* stacks;         // nb x ns x R x R
    const double* A0;             // nb x ns (nullptr: 0)
};

// What an evaluation leaves for the tangents, per slice (all nullptr: not kept).
struct CalKeep {
    double2* Q;   // D x D
    double2* E;   // W x W
    double* T;    // R x R
    double* Ts;   // R x R: d T / d sigma
    double* S;    // sum |T|
};

// Work areas of a cluster, in global memory (they stay in L2).
struct CalWork {
    double2* Q;  // D x D
    double2* S;  // W x D
    double2* E;  // W x W
    double2* X;  // D x W
    double* J;   // R x W
    double* dJ;  // R x W
    double* g;   // R x R: g_T
};

__host__ __device__ inline size_t cal_al(size_t v) { return (v + 255) / 256 * 256; }
__host__ __device__ inline size_t cal_work_bytes(int D, int W, int R) {
    return cal_al((size_t)D * D * 16) + 2 * cal_al((size_t)D * W * 16) + cal_al((size_t)W * W * 16) +
           2 * cal_al((size_t)R * W * 8) + cal_al((size_t)R * R * 8);
}

__device__ inline CalWork cal_carve(char* base, int D, int W, int R) {
    CalWork w;
    auto take = [&](size_t b) { char* q = base; base += cal_al(b); return q; };
    w.Q = (double2*)take((size_t)D * D * 16);
    w.S = (double2*)take((size_t)D * W * 16);
    w.E = (double2*)take((size_t)W * W * 16);
    w.X = (double2*)take((size_t)D * W * 16);
    w.J = (double*)take((size_t)R * W * 8);
    w.dJ = (double*)take((size_t)R * W * 8);
    w.g = (double*)take((size_t)R * R * 8);
    return w;
}

// Shared memory: reduction areas, transform buffer, a tile (pupil rows, or W rows of
// an intensity and R rows of V1 by LINES columns), and the transposed blur matrix where
// it fits; its derivative is read through L1.  With both in shared memory and 128
// registers two CTAs shared an SM; 85 registers spill next to nothing, and with three
// the latency-bound kernels take 1.84 and 0.25 ms (k_cal_tangent, k_cal_eval) instead of
// 2.07 and 0.28.
constexpr int CAL_RED_BYTES = 2048;
constexpr size_t CAL_G_SMEM = 32 * 1024;
__host__ __device__ inline size_t cal_tile_bytes(int N, int D, int W, int R) {
    const size_t lines = fl_lines(N), q = lines * (D | 1) * 16, x = (size_t)(W + R) * lines * 8;
    return cal_al(q > x ? q : x);
}
__host__ __device__ inline size_t cal_smem(int N, int D, int W, int R) {
    const size_t g = (size_t)W * R * 8;
    return CAL_RED_BYTES + FL_SMEM + cal_tile_bytes(N, D, W, R) + (g <= CAL_G_SMEM ? g : 0);
}

struct CalSmem {
    double* red;
    double2* buf;
    char* tile;
    const double *GT, *dGT;
};
template <int NFFT>
__device__ __forceinline__ CalSmem cal_begin(const CalView& V, char* smem) {
    CalSmem m{(double*)smem, (double2*)(smem + CAL_RED_BYTES), smem + CAL_RED_BYTES + FL_SMEM, V.GT, V.dGT};
    const int n = V.W * V.R;
    if ((size_t)n * 8 <= CAL_G_SMEM) {
        double* g = (double*)(m.tile + cal_tile_bytes(NFFT, V.D, V.W, V.R));
        for (int k = threadIdx.x; k < n; k += FL_THREADS) g[k] = V.GT[k];
        m.GT = g;
    }
    __syncthreads();
    return m;
}

// S (w, a) from pupil rows: field(a, b) gives the pupil field.  A CTA takes every
// step-th tile of LINES rows.
template <class F, class FIELD>
__device__ __forceinline__ void cal_rows(const CalView& V, const CalSmem& m, int first, int step, double2* S,
                                         const FIELD& field) {
    constexpr int N = F::N, L = F::LINES;
    const int D = V.D, DP = D | 1, W = V.W, a0 = V.a0;
    double2* Qt = (double2*)m.tile;
    for (int r0 = first * L; r0 < D; r0 += step * L) {
        for (int k = threadIdx.x; k < L * D; k += FL_THREADS) {
            const int l = k / D, b = k - l * D;
            Qt[l * DP + b] = r0 + l < D ? field(r0 + l, b) : make_double2(0, 0);
        }
        __syncthreads();
        auto ld = [&](unsigned k, unsigned l) {
            const int b = (int)k - a0;
            return (unsigned)b < (unsigned)D ? Qt[l * DP + b] : make_double2(0, 0);
        };
        auto st = [&](unsigned k, unsigned l, int, double2 v) {
            const unsigned o = (k + W / 2) & (N - 1);
            if (o < (unsigned)W && r0 + (int)l < D) S[(size_t)o * D + r0 + l] = v;
        };
        fl_transform<F, 1>(m.buf, V.tw, ld, st);
        __syncthreads();
    }
}

// Window columns: value(i, j, e) takes each E(i, j) and gives the intensity that is
// blurred along its first index into J (and by dG into dJ when it is not null).
template <class F, class VALUE>
__device__ __forceinline__ void cal_cols(const CalView& V, const CalSmem& m, int first, int step, const double2* S,
                                         double* J, double* dJ, const VALUE& value) {
    constexpr int N = F::N, L = F::LINES;
    const int D = V.D, W = V.W, R = V.R, a0 = V.a0;
    double* X = (double*)m.tile;
    for (int c0 = first * L; c0 < W; c0 += step * L) {
        auto ld = [&](unsigned k, unsigned l) {
            const int a = (int)k - a0;
            return (unsigned)a < (unsigned)D && c0 + (int)l < W ? S[(size_t)(c0 + l) * D + a] : make_double2(0, 0);
        };
        auto st = [&](unsigned k, unsigned l, int, double2 v) {
            const unsigned o = (k + W / 2) & (N - 1);
            if (o < (unsigned)W && c0 + (int)l < W) X[o * L + l] = value((int)o, c0 + (int)l, v);
        };
        fl_transform<F, 1>(m.buf, V.tw, ld, st);
        __syncthreads();
        blur_tile(m.GT, X, R, W, L, min(L, W), J + c0);
        if (dJ) blur_tile(m.dGT, X, R, W, L, min(L, W), dJ + c0);
        __syncthreads();
    }
}

// out(pixel, sum_j G[j'][j] J[i'][j] [+ sum_j G[j'][j] dJ.. ]) for rows i0 .. i1 - 1, two
// rows by two columns a thread.  SIGMA: sum_j dJ[i'][j] G[j'][j] + J[i'][j] dG[j'][j].
template <bool SIGMA, class OUT>
__device__ __forceinline__ void cal_second(const CalView& V, const CalSmem& m, const double* J, const double* dJ, int i0,
                                           int i1, const OUT& out) {
    const int W = V.W, R = V.R, hp = R / 2;
    for (int t = threadIdx.x; t < (i1 - i0) / 2 * hp; t += FL_THREADS) {
        const int ip = i0 + 2 * (t / hp), jp = 2 * (t % hp);
        const double *a = (SIGMA ? dJ : J) + (size_t)ip * W, *c = J + (size_t)ip * W;
        double s00 = 0, s01 = 0, s10 = 0, s11 = 0;
#pragma unroll 4
        for (int j = 0; j < W; j += 2) {
            const double2 x0 = *(const double2*)(a + j), x1 = *(const double2*)(a + W + j);
            const double2 g0 = *(const double2*)(m.GT + (size_t)j * R + jp), g1 = *(const double2*)(m.GT + (size_t)(j + 1) * R + jp);
            s00 = fma(x0.y, g1.x, fma(x0.x, g0.x, s00));
            s01 = fma(x0.y, g1.y, fma(x0.x, g0.y, s01));
            s10 = fma(x1.y, g1.x, fma(x1.x, g0.x, s10));
            s11 = fma(x1.y, g1.y, fma(x1.x, g0.y, s11));
            if (SIGMA) {
                const double2 y0 = *(const double2*)(c + j), y1 = *(const double2*)(c + W + j);
                const double2 d0 = *(const double2*)(m.dGT + (size_t)j * R + jp),
                              d1 = *(const double2*)(m.dGT + (size_t)(j + 1) * R + jp);
                s00 = fma(y0.y, d1.x, fma(y0.x, d0.x, s00));
                s01 = fma(y0.y, d1.y, fma(y0.x, d0.y, s01));
                s10 = fma(y1.y, d1.x, fma(y1.x, d0.x, s10));
                s11 = fma(y1.y, d1.y, fma(y1.x, d0.y, s11));
            }
        }
        out(ip * R + jp, s00);
        out(ip * R + jp + 1, s01);
        out((ip + 1) * R + jp, s10);
        out((ip + 1) * R + jp + 1, s11);
    }
}

// mode 0: NLL (+ model, psi), mode 1: NLL + adjoint.  One cluster per (bead, slice).
// out_slice: per slice NOUT values; gphi: per slice the phase gradient, [b][a]; K: per
// slice what the tangents need.  305 slices of 32 px, 45 modes, N = 128: 248 us (mode 1),
// bound by the latency of its passes and barriers (111 clusters at once); the direct sums
// with one output a thread, read from the work area, took 993 us.
template <int NFFT>
__global__ void __launch_bounds__(FL_THREADS, 3) k_cal_eval(CalView V, const double* phase, const double* bead, int mode,
                                                            CalKeep K, char* scratch, size_t per_cluster,
                                                            double* out_slice, double* gphi, double* model,
                                                            double* psi_out) {
    extern __shared__ __align__(256) char cal_sm[];
    using F = FftLines<NFFT>;
    constexpr int N = F::N, L = F::LINES;
    const int D = V.D, W = V.W, R = V.R, RR = R * R, tid = threadIdx.x;
    const Cluster cl;
    const CalSmem m = cal_begin<NFFT>(V, cal_sm);
    double *part1 = m.red + 128, *part9 = m.red + 136, *part4 = m.red + 152;  // sums of 1, 9 and 4 values
    CalWork w = cal_carve(scratch + cl.id() * per_cluster, D, W, R);
    const int i0 = cl.row0(R), i1 = cl.row1(R), nt = (i1 - i0) * R, px0 = i0 * R;
    // T of the CTA's rows: in the transform buffer until the adjoint needs it, else in w.g
    double* T = (size_t)2 * nt * 8 <= FL_SMEM ? (double*)m.buf : nullptr;
    for (int bs = cl.id(); bs < V.nb * V.ns; bs += cl.count()) {
        const int b = bs / V.ns, s = bs % V.ns;
        const double* th = bead + (size_t)b * V.pb;
        const double x = th[0], y = th[1], zoil = V.dz[s] + th[2];
        const double At = (V.A0 ? V.A0[bs] : 0.0) + th[3 + s];
        const double* c = th + 3 + V.ns;
        double2* Q = K.Q ? K.Q + (size_t)bs * D * D : w.Q;
        double2* E = K.E ? K.E + (size_t)bs * W * W : w.E;
        cal_rows<F>(V, m, cl.rank, cl.size, w.S, [&](int a, int bb) {
            const int k = a * D + bb;
            const double p = V.pupil[k];
            double2 q = make_double2(0, 0);
            if (p != 0) {
                double sn, cs;
                sincos(phase[k] + V.kx[a] * x + V.ky[bb] * y - V.kzoil[k] * zoil, &sn, &cs);
                q = make_double2(p * cs, p * sn);
            }
            Q[k] = q;
            return q;
        });
        cl.sync();
        cal_cols<F>(V, m, cl.rank, cl.size, w.S, w.J, mode == 1 ? w.dJ : nullptr, [&](int i, int j, double2 e) {
            if (mode == 1) E[(size_t)i * W + j] = e;
            return e.x * e.x + e.y * e.y;
        });
        cl.sync();
        double* Tp = T ? T : w.g + px0;  // (the rows of w.g are the CTA's own until g_T is complete)
        double sum[1] = {0};
        cal_second<false>(V, m, w.J, nullptr, i0, i1, [&](int px, double v) {
            Tp[px - px0] = v;
            sum[0] += fabs(v);
            if (K.T) K.T[(size_t)bs * RR + px] = v;
        });
        cluster_sum<1>(cl, sum, m.red, part1);
        const double Ssum = sum[0];
        const double* d = V.stacks + (size_t)bs * RR;
        double acc[9];  // nll, d/da, d/dc[6], sum g_psi psi
#pragma unroll
        for (int q = 0; q < 9; ++q) acc[q] = 0.0;
        auto weight = [&](int k, double psi, double* mu_) {  // 1 - d / mu, 0 where mu is clamped
            const int i = k / R, ii = k - i * R;
            double bg = 0;
#pragma unroll
            for (int q = 0; q < NPOLY; ++q) bg += c[q] * poly_m(q, i, ii);
            const double raw = psi * At + bg;
            *mu_ = raw <= 0 ? 0.00000001 : raw;
            return raw <= 0 ? 0.0 : 1.0 - d[k] / *mu_;
        };
        for (int t = tid; t < nt; t += FL_THREADS) {
            const int k = px0 + t, i = k / R, ii = k - i * R;
            const double psi = fabs(Tp[t]) / Ssum;
            double mu;
            const double wgt = weight(k, psi, &mu);
            acc[0] += mu - d[k] * log(mu);
            if (model) model[(size_t)bs * RR + k] = mu;
            if (psi_out) psi_out[(size_t)bs * RR + k] = psi;
            acc[1] += wgt * psi;
#pragma unroll
            for (int q = 0; q < NPOLY; ++q) acc[2 + q] += wgt * poly_m(q, i, ii);
            acc[8] += At * wgt * psi;
        }
        cluster_sum<9>(cl, acc, m.red, part9);
        double tot4[4] = {0, 0, 0, 0};  // d/dsigma, d/dx, d/dy, d/dz
        if (mode == 1) {
            // g_T = sgn(T) (g_psi - sum g_psi psi) / S, and its product with dT / dsigma
            double* gs = (double*)m.tile;  // (a thread keeps its own pixels' g_T for the product)
            const bool own = (size_t)nt * 8 <= cal_tile_bytes(N, D, W, R);
            for (int t = tid; t < nt; t += FL_THREADS) {
                const double tv = Tp[t], psi = fabs(tv) / Ssum;
                double mu;
                const double g = (tv < 0 ? -1.0 : 1.0) * (At * weight(px0 + t, psi, &mu) - acc[8]) / Ssum;
                w.g[px0 + t] = g;
                if (own) gs[t] = g;
            }
            __syncthreads();
            cal_second<true>(V, m, w.J, w.dJ, i0, i1, [&](int px, double v) {
                tot4[0] += (own ? gs[px - px0] : w.g[px]) * v;
                if (K.Ts) K.Ts[(size_t)bs * RR + px] = v;
            });
            cl.sync();
            // columns: V1 = g_T G, g_I = G^T V1, X = C^H (g_I o E)
            double* gI = (double*)m.tile;             // [i][column]
            double* V1 = gI + (size_t)W * L;          // [i'][column]
            for (int c0 = cl.rank * L; c0 < W; c0 += cl.size * L) {
                const int cols = min(L, W);
                for (int t = tid; t < R * cols; t += FL_THREADS) {
                    const int ip = t / cols, l = t - ip * cols;
                    const double *g = w.g + (size_t)ip * R, *gt = m.GT + (size_t)(c0 + l) * R;
                    double v = 0;
#pragma unroll 4
                    for (int jp = 0; jp < R; ++jp) v = fma(g[jp], gt[jp], v);
                    V1[ip * L + l] = v;
                }
                __syncthreads();
                for (int t = tid; t < W / 2 * (cols / 2); t += FL_THREADS) {
                    const int i = 2 * (t / (cols / 2)), l = 2 * (t % (cols / 2));
                    const double *g0 = m.GT + (size_t)i * R, *g1 = g0 + R;
                    double s00 = 0, s01 = 0, s10 = 0, s11 = 0;
#pragma unroll 2
                    for (int ip = 0; ip < R; ip += 2) {
                        const double2 p0 = *(const double2*)(g0 + ip), p1 = *(const double2*)(g1 + ip);
                        const double2 v0 = *(const double2*)(V1 + ip * L + l), v1 = *(const double2*)(V1 + (ip + 1) * L + l);
                        s00 = fma(p0.y, v1.x, fma(p0.x, v0.x, s00));
                        s01 = fma(p0.y, v1.y, fma(p0.x, v0.y, s01));
                        s10 = fma(p1.y, v1.x, fma(p1.x, v0.x, s10));
                        s11 = fma(p1.y, v1.y, fma(p1.x, v0.y, s11));
                    }
                    gI[i * L + l] = s00; gI[i * L + l + 1] = s01;
                    gI[(i + 1) * L + l] = s10; gI[(i + 1) * L + l + 1] = s11;
                }
                __syncthreads();
                auto ld = [&](unsigned k, unsigned l) {
                    const unsigned o = (k + W / 2) & (N - 1);
                    if (o >= (unsigned)W || c0 + (int)l >= W) return make_double2(0, 0);
                    const double2 e = E[(size_t)o * W + c0 + l];
                    const double g = gI[o * L + l];
                    return make_double2(g * e.x, g * e.y);
                };
                auto st = [&](unsigned k, unsigned l, int, double2 v) {
                    const int a = (int)k - V.a0;
                    if ((unsigned)a < (unsigned)D && c0 + (int)l < W) w.X[(size_t)a * W + c0 + l] = v;
                };
                fl_transform<F, -1>(m.buf, V.tw, ld, st);
                __syncthreads();
            }
            cl.sync();
            // rows: Qbar = X conj(C), g_phi = 2 Im(conj(Q) Qbar) and its registration sums
            double* gp = gphi + (size_t)bs * D * D;
            for (int r0 = cl.rank * L; r0 < D; r0 += cl.size * L) {
                auto ld = [&](unsigned k, unsigned l) {
                    const unsigned o = (k + W / 2) & (N - 1);
                    return o < (unsigned)W && r0 + (int)l < D ? w.X[(size_t)(r0 + l) * W + o] : make_double2(0, 0);
                };
                auto st = [&](unsigned k, unsigned l, int, double2 v) {
                    const int bb = (int)k - V.a0, a = r0 + (int)l;
                    if ((unsigned)bb >= (unsigned)D || a >= D) return;
                    const double2 q = Q[(size_t)a * D + bb];
                    const double g = 2.0 * (q.x * v.y - q.y * v.x);
                    gp[(size_t)bb * D + a] = g;
                    tot4[1] += g * V.kx[a];
                    tot4[2] += g * V.ky[bb];
                    tot4[3] -= g * V.kzoil[(size_t)a * D + bb];
                };
                fl_transform<F, -1>(m.buf, V.tw, ld, st);
                __syncthreads();
            }
            cluster_sum<4>(cl, tot4, m.red, part4);
        }
        if (cl.rank == 0 && tid == 0) {
            double* o = out_slice + (size_t)NOUT * bs;
            o[0] = acc[0]; o[1] = acc[1]; o[2] = tot4[0];
            for (int q = 0; q < NPOLY; ++q) o[3 + q] = acc[2 + q];
            for (int q = 0; q < 3; ++q) o[3 + NPOLY + q] = tot4[1 + q];
            if (K.S) K.S[bs] = Ssum;
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may read its shared memory
}

// Tangent maps d mu / d theta_u of every slice: u < nzr Zernike modes 3 .. (Z: basis),
// then sigma, x, y, z.  Items are (u, slice), a CTA each, from the fields that the
// evaluation kept.  tan: per (u, bs) R x R.  46 directions x 305 slices of 32 px (N = 128):
// 1.8 ms, bound by latency as k_cal_eval; repeating the forward model per direction with
// direct sums took 30.3 ms.
template <int NFFT>
__global__ void __launch_bounds__(FL_THREADS, 3) k_cal_tangent(CalView V, CalKeep K, const double* bead, const double* Z,
                                                               int nzr, char* scratch, size_t per_cta, double* tan) {
    extern __shared__ __align__(256) char cal_sm[];
    using F = FftLines<NFFT>;
    const int D = V.D, W = V.W, R = V.R, RR = R * R, nbs = V.nb * V.ns, tid = threadIdx.x;
    const Cluster cl;  // of one CTA
    const CalSmem m = cal_begin<NFFT>(V, cal_sm);
    CalWork w = cal_carve(scratch + blockIdx.x * per_cta, D, W, R);
    double* aux = (size_t)RR * 8 <= FL_SMEM ? (double*)m.buf : w.g;  // sgn(T) dT
    for (int item = blockIdx.x; item < (nzr + 4) * nbs; item += gridDim.x) {
        const int u = item / nbs, bs = item - u * nbs, b = bs / V.ns, s = bs - b * V.ns;
        const double* T = K.T + (size_t)bs * RR;
        double dsum[1] = {0};
        if (u == nzr) {
            for (int k = tid; k < RR; k += FL_THREADS) {
                const double v = (T[k] < 0 ? -1.0 : 1.0) * K.Ts[(size_t)bs * RR + k];
                aux[k] = v;
                dsum[0] += v;
            }
        } else {
            const double2* Q = K.Q + (size_t)bs * D * D;
            const double2* E = K.E + (size_t)bs * W * W;
            const double* Zu = Z + (size_t)(u < nzr ? u + 3 : 0) * D * D;
            cal_rows<F>(V, m, 0, 1, w.S, [&](int a, int bb) {  // i Q dphi
                const double2 q = Q[a * D + bb];
                const double p = u < nzr ? Zu[a * D + bb] : u == nzr + 1 ? V.kx[a] : u == nzr + 2 ? V.ky[bb] : -V.kzoil[a * D + bb];
                return make_double2(-q.y * p, q.x * p);
            });
            cal_cols<F>(V, m, 0, 1, w.S, w.J, nullptr, [&](int i, int j, double2 e) {
                const double2 e0 = E[(size_t)i * W + j];
                return 2.0 * (e0.x * e.x + e0.y * e.y);
            });
            cal_second<false>(V, m, w.J, nullptr, 0, R, [&](int px, double v) {
                v = (T[px] < 0 ? -1.0 : 1.0) * v;
                aux[px] = v;
                dsum[0] += v;
            });
        }
        cluster_sum<1>(cl, dsum, m.red, m.red + 128);
        const double At = (V.A0 ? V.A0[bs] : 0.0) + bead[(size_t)b * V.pb + 3 + s], S = K.S[bs];
        double* out = tan + ((size_t)u * nbs + bs) * RR;
        for (int k = tid; k < RR; k += FL_THREADS) out[k] = At * (aux[k] - fabs(T[k]) / S * dsum[0]) / S;
        __syncthreads();
    }
}

// Per-slice Gauss-Newton blocks sum_p J_u J_v / mu over the slice's local
// directions: the nzr + 4 tangents, then psi (for a_bs) and the NPOLY background
// monomials; clamped pixels contribute nothing.  gram: per slice nl (nl + 1) / 2
// entries (upper triangle, row-major).
// 32 pixels of every direction are staged pixel by pixel in shared memory; a thread
// owns a 4 x 4 block of entries (eight 8-byte values in four loads for 16 FMAs) over
// half of the pixels.  53 directions x 305 slices of 32 px: 255 us; one entry a thread
// and product took 1.42 ms.
constexpr int GN_CHUNK = 32;
__host__ __device__ inline int gn_stride(int nl) { return (nl + 3) / 4 * 4 + 2; }
__global__ void __launch_bounds__(FL_THREADS) k_cal_gn(CalView V, int nzr, const double* tan, const double* model,
                                                       const double* psi, double* gram) {
    extern __shared__ __align__(16) double gn_sm[];
    const int R = V.R, RR = R * R, nbs = V.nb * V.ns, nt = nzr + 4, nl = nt + 1 + NPOLY, ne = nl * (nl + 1) / 2;
    const int nt4 = (nl + 3) / 4, LS = gn_stride(nl), tiles = nt4 * (nt4 + 1) / 2;
    constexpr int HALF = FL_THREADS / 2;
    double* Lm = gn_sm;                             // [pixel][direction]
    double* inv = Lm + (size_t)GN_CHUNK * LS;       // 1 / mu
    double* other = inv + GN_CHUNK;                 // [16][HALF]: the second half's sums
    const int half = threadIdx.x / HALF, lane = threadIdx.x % HALF;
    for (int bs = blockIdx.x; bs < nbs; bs += gridDim.x)
        for (int t0 = 0; t0 < tiles; t0 += HALF) {
            int tu = 0, tv = t0 + lane;
            const bool act = tv < tiles;
            while (act && tv >= nt4 - tu) { tv -= nt4 - tu; ++tu; }
            tv += tu;
            const int u0 = act ? 4 * tu : 0, v0 = act ? 4 * tv : 0;
            double acc[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) acc[q] = 0;
            for (int p0 = 0; p0 < RR; p0 += GN_CHUNK) {
                __syncthreads();
                for (int k = threadIdx.x; k < 4 * nt4 * GN_CHUNK; k += FL_THREADS) {
                    const int u = k / GN_CHUNK, pp = k % GN_CHUNK, p = p0 + pp;
                    double v = 0;
                    if (p < RR && u < nl) {
                        if (u < nt) v = tan[((size_t)u * nbs + bs) * RR + p];
                        else if (u == nt) v = psi[(size_t)bs * RR + p];
                        else v = poly_m(u - nt - 1, p / R, p % R);
                    }
                    Lm[pp * LS + u] = v;
                }
                for (int pp = threadIdx.x; pp < GN_CHUNK; pp += FL_THREADS) {
                    const double mu = p0 + pp < RR ? model[(size_t)bs * RR + p0 + pp] : 0.0;
                    inv[pp] = mu > 0.00000001 ? 1.0 / mu : 0.0;
                }
                __syncthreads();
#pragma unroll 2
                for (int pp = half * (GN_CHUNK / 2); pp < (half + 1) * (GN_CHUNK / 2); ++pp) {
                    const double* r = Lm + pp * LS;
                    const double iv = inv[pp];
                    const double2 a0 = *(const double2*)(r + u0), a1 = *(const double2*)(r + u0 + 2);
                    const double2 c0 = *(const double2*)(r + v0), c1 = *(const double2*)(r + v0 + 2);
                    const double a[4] = {a0.x * iv, a0.y * iv, a1.x * iv, a1.y * iv}, c[4] = {c0.x, c0.y, c1.x, c1.y};
#pragma unroll
                    for (int q = 0; q < 16; ++q) acc[q] = fma(a[q / 4], c[q % 4], acc[q]);
                }
            }
            __syncthreads();
            if (half == 1) {
#pragma unroll
                for (int q = 0; q < 16; ++q) other[q * HALF + lane] = acc[q];
            }
            __syncthreads();
            if (half == 0 && act) {
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const int u = u0 + q / 4, v = v0 + q % 4;
                    if (u <= v && v < nl)
                        gram[(size_t)bs * ne + (size_t)u * nl - (size_t)u * (u - 1) / 2 + (v - u)] = acc[q] + other[q * HALF + lane];
                }
            }
        }
}

// Pupil phase sum_{i >= 3} a_i Z_i, in the order of the modes.
__global__ void k_cal_phase(const double* Z, const double* coef, int nz, int DD, double* phase) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= DD) return;
    double s = 0;
    for (int i = 3; i < nz; ++i) s = __dadd_rn(s, __dmul_rn(coef[i], Z[(size_t)i * DD + k]));
    phase[k] = s;
}

// Phase gradient of the whole stack: the slices' [b][a] maps summed in a fixed order
// (eight groups of slices, then the groups) into [a][b].
__global__ void __launch_bounds__(256) k_cal_gsum(const double* gphi, int nbs, int D, double* gsum) {
    __shared__ double part[8][32];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31, k = blockIdx.x * 32 + lane, DD = D * D;
    double s = 0;
    if (k < DD)
#pragma unroll 4
        for (int bs = g; bs < nbs; bs += 8) s += gphi[(size_t)bs * DD + k];
    part[g][lane] = s;
    __syncthreads();
    if (g == 0 && k < DD) {
        s = 0;
        for (int q = 0; q < 8; ++q) s += part[q][lane];
        gsum[(k % D) * D + k / D] = s;
    }
}

// The gradient: CTA i < nz projects gsum on mode i (0 for i < 3); CTA nz + b forms
// bead b's (x, y, z, a_0 .., c_0 ..); the last CTA the totals (nll, d/dsigma).
// res = tot(2) | gz(nz) | gb(nb x pb).  modes = 0: the totals only.
__global__ void __launch_bounds__(256) k_cal_finish(CalView V, const double* out_slice, const double* gsum, const double* Z,
                                                    int nz, double* res) {
    __shared__ double red[8];
    const int nbs = V.nb * V.ns, DD = V.D * V.D, job = blockIdx.x;
    auto total = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        __syncthreads();
        double s = 0;
        for (int q = 0; q < 8; ++q) s += red[q];
        return s;
    };
    auto slices = [&](int first, int n, int col) {
        double v = 0;
        for (int k = threadIdx.x; k < n; k += 256) v += out_slice[(size_t)NOUT * (first + k) + col];
        return total(v);
    };
    if (job == (int)gridDim.x - 1) {
        const double a = slices(0, nbs, 0), c = slices(0, nbs, 2);
        if (threadIdx.x == 0) { res[0] = a; res[1] = c; }
    } else if (job < nz) {
        double v = 0;
        if (job >= 3)
            for (int k = threadIdx.x; k < DD; k += 256) v += gsum[k] * Z[(size_t)job * DD + k];
        v = total(v);
        if (threadIdx.x == 0) res[2 + job] = v;
    } else {
        const int b = job - nz;
        double* o = res + 2 + nz + (size_t)b * V.pb;
        for (int q = 0; q < 3 + NPOLY; ++q) {
            const double v = slices(b * V.ns, V.ns, q < 3 ? 3 + NPOLY + q : q);
            if (threadIdx.x == 0) o[q < 3 ? q : V.ns + q] = v;
        }
        for (int s = threadIdx.x; s < V.ns; s += 256) o[3 + s] = out_slice[(size_t)NOUT * (b * V.ns + s) + 1];
    }
}

// The parameter vector theta = (modes 3 .., [sigma], per bead x, y, z, a_s, c_k): the
// bead, slice (-1: any) and local Gram direction of index p.
struct CalTheta {
    int bead, slice, u;
};
__device__ inline CalTheta cal_theta(const CalView& V, int nzr, int fit_sigma, int p) {
    if (p < nzr) return {-1, -1, p};
    const int boff = nzr + (fit_sigma ? 1 : 0);
    if (p < boff) return {-1, -1, nzr};
    const int b = (p - boff) / V.pb, q = p - boff - b * V.pb;
    if (q < 3) return {b, -1, nzr + 1 + q};
    if (q < 3 + V.ns) return {b, q - 3, nzr + 4};
    return {b, -1, nzr + 5 + (q - 3 - V.ns)};
}

// Gauss-Newton matrix H (npar x npar, both triangles) from the slices' blocks, a thread
// an entry, slices in order.
__global__ void k_cal_hess(CalView V, int nzr, int fit_sigma, int npar, const double* gram, double* H) {
    const int p = blockIdx.y * blockDim.y + threadIdx.y, q = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npar || q >= npar || q < p) return;
    const CalTheta a = cal_theta(V, nzr, fit_sigma, p), c = cal_theta(V, nzr, fit_sigma, q);
    const int nl = nzr + 5 + NPOLY, ne = nl * (nl + 1) / 2, u = min(a.u, c.u), v = max(a.u, c.u);
    const int bead = max(a.bead, c.bead), slice = max(a.slice, c.slice);
    double s = 0;
    if ((a.bead < 0 || c.bead < 0 || a.bead == c.bead) && (a.slice < 0 || c.slice < 0 || a.slice == c.slice)) {
        const int s0 = slice >= 0 ? bead * V.ns + slice : bead >= 0 ? bead * V.ns : 0;
        const int s1 = slice >= 0 ? s0 + 1 : bead >= 0 ? s0 + V.ns : V.nb * V.ns;
        const double* g = gram + (size_t)u * nl - (size_t)u * (u - 1) / 2 + (v - u);
#pragma unroll 4
        for (int bs = s0; bs < s1; ++bs) s += g[(size_t)bs * ne];
    }
    H[(size_t)p * npar + q] = s;
    H[(size_t)q * npar + p] = s;
}

// Damped solve (H + lambda max(diag H, 1e-12)) x = -g.  The beads' parameters couple only
// through the ng shared ones (modes and sigma), so a CTA a bead eliminates its pb
// parameters (k_cal_bead), one CTA solves for the shared ones (k_cal_shared), and a CTA a
// bead takes its own from them (k_cal_back).  45 modes and 5 beads of 61 slices, 393
// parameters: 314 us; one factorisation of the whole matrix by one CTA, which fills the
// blocks between beads, took 1270.
//
// The pieces are blocked Cholesky factorisations by one CTA: 32 columns at a time, the
// diagonal block by one warp with a row in a lane's registers, the panel a row a thread,
// the trailing matrix in 4 x 4 blocks from panels staged in shared memory.
constexpr int CH_B = 32, CH_THREADS = 512, CH_ROWS = 256;
constexpr int CH_SMEM = (CH_B * (CH_B + 1) + 2 * CH_ROWS * (CH_B + 2)) * 8 + 64;

// Eliminates the first n columns of the lower triangle of A (rows x cols, row stride ld):
// the factor in their place, the Schur complement in rows and columns n .. .  False when
// a pivot is not positive.
__device__ bool chol(double* A, int ld, int n, int rows, int cols, double* ch_sm) {
    double* dg = ch_sm;                   // [32][33]: the diagonal block
    double* pa = dg + CH_B * (CH_B + 1);  // panel rows of the block rows, [row][34]
    double* pc = pa + CH_ROWS * (CH_B + 2);  // panel rows of the block columns
    int* bad = (int*)(pc + CH_ROWS * (CH_B + 2));
    constexpr int PS = CH_B + 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) *bad = 0;
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += CH_B) {
        const int nb = min(CH_B, n - k0);
        if (warp == 0) {
            double r[CH_B];
#pragma unroll
            for (int j = 0; j < CH_B; ++j)
                r[j] = j < nb && lane < nb && j <= lane ? A[(size_t)(k0 + lane) * ld + k0 + j] : 0.0;
            bool fine = true;
#pragma unroll
            for (int j = 0; j < CH_B; ++j) {
                if (j >= nb) break;
                const double piv = __shfl_sync(0xffffffffu, r[j], j);
                if (!(piv > 0)) { fine = false; break; }
                const double d = sqrt(piv);
                r[j] = lane == j ? d : r[j] / d;
#pragma unroll
                for (int k = j + 1; k < CH_B; ++k) {
                    const double c = __shfl_sync(0xffffffffu, r[j], k);
                    if (lane >= k) r[k] -= r[j] * c;
                }
            }
#pragma unroll
            for (int j = 0; j < CH_B; ++j) dg[lane * (CH_B + 1) + j] = r[j];
            if (!fine && lane == 0) *bad = 1;
        }
        __syncthreads();
        if (*bad) return false;
        for (int k = tid; k < nb * nb; k += CH_THREADS) {
            const int i = k / nb, j = k - i * nb;
            if (j <= i) A[(size_t)(k0 + i) * ld + k0 + j] = dg[i * (CH_B + 1) + j];
        }
        for (int i = k0 + nb + tid; i < rows; i += CH_THREADS) {  // the panel below it
            double r[CH_B];
            double* a = A + (size_t)i * ld + k0;
#pragma unroll
            for (int j = 0; j < CH_B; ++j) r[j] = j < nb ? a[j] : 0.0;
#pragma unroll
            for (int j = 0; j < CH_B; ++j) {
                if (j >= nb) break;
                double s = r[j];
#pragma unroll
                for (int k = 0; k < j; ++k) s -= r[k] * dg[j * (CH_B + 1) + k];
                r[j] = s / dg[j * (CH_B + 1) + j];
                a[j] = r[j];
            }
        }
        __syncthreads();
        // trailing rows i >= k0 + nb, columns k0 + nb <= j <= i (and j < cols)
        for (int i0 = k0 + nb; i0 < rows; i0 += CH_ROWS)
            for (int j0 = k0 + nb; j0 <= i0 + CH_ROWS - 1 && j0 < cols; j0 += CH_ROWS) {
                const int ni = min(CH_ROWS, rows - i0), nj = min(CH_ROWS, cols - j0);
                __syncthreads();
                for (int k = tid; k < CH_ROWS * CH_B; k += CH_THREADS) {
                    const int i = k / CH_B, j = k % CH_B;
                    pa[i * PS + j] = i < ni && j < nb ? A[(size_t)(i0 + i) * ld + k0 + j] : 0.0;
                    if (j0 != i0) pc[i * PS + j] = i < nj && j < nb ? A[(size_t)(j0 + i) * ld + k0 + j] : 0.0;
                }
                __syncthreads();
                const double* pj = j0 == i0 ? pa : pc;
                const int bi = (ni + 3) / 4, bj = (nj + 3) / 4;
                for (int t = tid; t < bi * bj; t += CH_THREADS) {
                    const int i = t / bj * 4, j = t % bj * 4;
                    if (j0 + j > i0 + i + 3) continue;
                    double s[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) s[q] = 0;
#pragma unroll 4
                    for (int k = 0; k < CH_B; k += 2) {
                        double2 a[4], c[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            a[q] = *(const double2*)(pa + (i + q) * PS + k);
                            c[q] = *(const double2*)(pj + (j + q) * PS + k);
                        }
#pragma unroll
                        for (int q = 0; q < 16; ++q) s[q] = fma(a[q / 4].y, c[q % 4].y, fma(a[q / 4].x, c[q % 4].x, s[q]));
                    }
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        const int ii = i + q / 4, jj = j + q % 4;
                        if (ii < ni && jj < nj && j0 + jj <= i0 + ii) A[(size_t)(i0 + ii) * ld + j0 + jj] -= s[q];
                    }
                }
            }
        __syncthreads();
    }
    return true;
}

// x = L^-T y, block by block: L the factor of n columns in A, y is overwritten.
__device__ void chol_back(const double* A, int ld, int n, double* y, double* x, double* ch_sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k1 = n; k1 > 0;) {
        const int k0 = (k1 - 1) / CH_B * CH_B, nb = k1 - k0;
        if (warp == 0) {
            double v = lane < nb ? y[k0 + lane] : 0.0;
            for (int j = nb - 1; j >= 0; --j) {
                const double xj = __shfl_sync(0xffffffffu, v, j) / A[(size_t)(k0 + j) * ld + k0 + j];
                if (lane == j) v = xj;
                else if (lane < j) v -= A[(size_t)(k0 + j) * ld + k0 + lane] * xj;
            }
            if (lane < nb) { ch_sm[lane] = v; x[k0 + lane] = v; }
        }
        __syncthreads();
        for (int i = tid; i < k0; i += CH_THREADS) {
            double v = y[i];
            for (int j = 0; j < nb; ++j) v -= A[(size_t)(k0 + j) * ld + i] * ch_sm[j];
            y[i] = v;
        }
        __syncthreads();
        k1 = k0;
    }
}

// Bead blockIdx.x: its block of H, the shared parameters' rows and -g as rows below
// (M = pb + ng + 1 of stride M), eliminated.  flags[0]: every pivot was positive.
__global__ void __launch_bounds__(CH_THREADS) k_cal_bead(const double* H, const double* g, int n, int ng, int pb,
                                                         double lambda, double* A, int* flags) {
    extern __shared__ __align__(16) double ch_sm[];
    const int M = pb + ng + 1, o = ng + blockIdx.x * pb;
    A += (size_t)blockIdx.x * M * M;
    for (int k = threadIdx.x; k < M * M; k += CH_THREADS) {
        const int i = k / M, j = k - i * M;
        if (j > i) continue;
        double v = 0.0;
        if (j < pb) v = i < pb ? H[(size_t)(o + i) * n + o + j] : i < M - 1 ? H[(size_t)(i - pb) * n + o + j] : -g[o + j];
        if (i == j && i < pb) v += lambda * fmax(v, 1e-12);
        A[k] = v;
    }
    __syncthreads();
    if (!chol(A, M, pb, M, M - 1, ch_sm) && threadIdx.x == 0) atomicAnd(flags, 0);
}

// The shared parameters: their block of H plus the beads' Schur complements.  S: (ng + 1) x
// ng work space.
__global__ void __launch_bounds__(CH_THREADS) k_cal_shared(const double* H, const double* g, int n, int ng, int pb, int nb,
                                                           double lambda, const double* A, double* S, double* x, int* flags) {
    extern __shared__ __align__(16) double ch_sm[];
    if (!*flags) return;
    const int M = pb + ng + 1;
    for (int k = threadIdx.x; k < (ng + 1) * ng; k += CH_THREADS) {
        const int i = k / ng, j = k - i * ng;
        if (j > i) continue;
        double v = i < ng ? H[(size_t)i * n + j] : -g[j];
        if (i == j) v += lambda * fmax(v, 1e-12);
        for (int b = 0; b < nb; ++b) v += A[(size_t)b * M * M + (size_t)(pb + i) * M + pb + j];
        S[k] = v;
    }
    __syncthreads();
    if (!chol(S, ng, ng, ng + 1, ng, ch_sm)) {
        if (threadIdx.x == 0) *flags = 0;
        return;
    }
    chol_back(S, ng, ng, S + (size_t)ng * ng, x, ch_sm);
}

__global__ void __launch_bounds__(CH_THREADS) k_cal_back(int ng, int pb, double* A, double* x, const int* flags) {
    extern __shared__ __align__(16) double ch_sm[];
    if (!*flags) return;
    const int M = pb + ng + 1;
    A += (size_t)blockIdx.x * M * M;
    double* y = A + (size_t)(M - 1) * M;
    for (int j = threadIdx.x; j < pb; j += CH_THREADS) {
        double v = y[j];
        for (int i = 0; i < ng; ++i) v -= A[(size_t)(pb + i) * M + j] * x[i];
        y[j] = v;
    }
    __syncthreads();
    chol_back(A, M, pb, y, x + ng + blockIdx.x * pb, ch_sm);
}

}  // namespace zola

// --------------------------------------------------------------------- host --
using namespace zola;

namespace {

double fact(int n) {
    double f = 1;
    for (int i = 2; i <= n; ++i) f *= i;
    return f;
}

double zern(int n, int m, double th, double rho) {
    int am = m < 0 ? -m : m;
    double s = 0;
    for (int k = 0; k <= (n - am) / 2; ++k)
        s += (((k & 1) ? -1.0 : 1.0) * fact(n - k)) / (fact(k) * fact((n + am) / 2 - k) * fact((n - am) / 2 - k)) *
             std::pow(rho, n - 2 * k);
    return m >= 0 ? s * std::cos(th * am) : s * std::sin(th * am);
}

// Zernike basis on the disk square for modes 0..nz-1 (optics.cpp's polynomial), on the
// device, kept with the PSF for the last nz.
cudaError_t basis(zola_psf* p, int nz) {
    if (p->d_calZ && p->cal_nz == nz) return cudaSuccess;
    if (p->d_calZ) cudaFree(p->d_calZ);
    p->d_calZ = nullptr;
    const int D = p->D, N = p->N;
    const double cc = (double)(N / 2) - 0.5;
    const double radius = (p->o.na / p->o.wavelength) * (N * p->o.xystep);
    std::vector<double> Z((size_t)nz * D * D, 0.0);
    std::vector<int> zn(nz), zm(nz);
    for (int idx = 0, n = 0; idx < nz; ++n)
        for (int m = -n; m <= n && idx < nz; m += 2, ++idx) { zn[idx] = n; zm[idx] = m; }
    for (int a = 0; a < D; ++a)
        for (int b = 0; b < D; ++b) {
            if (p->pupil[(size_t)a * D + b] == 0) continue;
            const double x = (p->a0 + a - cc) / radius, y = (p->a0 + b - cc) / radius;
            const double rho = std::sqrt(x * x + y * y), th = std::atan2(y, x);
            for (int i = 0; i < nz; ++i) Z[((size_t)i * D + a) * D + b] = rho < 1 ? zern(zn[i], zm[i], th, rho) : 0.0;
        }
    cudaError_t e = cudaMalloc(&p->d_calZ, Z.size() * 8);
    if (e == cudaSuccess) e = cudaMemcpy(p->d_calZ, Z.data(), Z.size() * 8, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {  // (nothing half made is kept)
        if (p->d_calZ) cudaFree(p->d_calZ);
        p->d_calZ = nullptr;
    }
    p->cal_nz = nz;
    return e;
}

struct CalRun {
    CalView V{};
    CalKeep K{};
    int nz = 0, N = 0;
    size_t per_cluster = 0;
    double *d_par = nullptr;   // coefficients | bead parameters | GT | dGT (uploaded per evaluation)
    double *d_res = nullptr;   // totals | d/dz_i | bead gradients
    double *d_phase = nullptr, *d_slice = nullptr, *d_gphi = nullptr, *d_gsum = nullptr, *d_stacks = nullptr,
           *d_const = nullptr;  // dz | A0
    char* scratch = nullptr;
    std::vector<double> par, res;
    double sigma = -1;
    size_t n_bead() const { return (size_t)V.nb * V.pb; }
    size_t head() const { return (nz + n_bead() + 1) / 2 * 2; }  // GT and dGT are read as pairs
};

// Carve the buffers q[k] (bytes[k] each, 256-byte aligned) from a grow-only
// device area of the context; repeated calls of the same size allocate nothing.
cudaError_t carve(void** area, size_t* cap, void** const* q, const size_t* bytes, int n) {
    size_t total = 0;
    for (int k = 0; k < n; ++k) total += cal_al(bytes[k]);
    if (total > *cap) {
        if (*area) {
            cudaDeviceSynchronize();
            cudaFree(*area);
            *area = nullptr;
            *cap = 0;
        }
        cudaError_t e = cudaMalloc(area, total);
        if (e != cudaSuccess) return e;
        *cap = total;
    }
    char* base = (char*)*area;
    for (int k = 0; k < n; ++k) {
        *q[k] = bytes[k] ? base : nullptr;
        base += cal_al(bytes[k]);
    }
    return cudaSuccess;
}

int cal_cuda(zola_ctx* ctx, cudaError_t e) {
    if (e == cudaSuccess) return ZOLA_OK;
    ctx->err = std::string("calibration: ") + cudaGetErrorString(e);
    return ZOLA_E_CUDA;
}

constexpr int CAL_CLUSTERS = 592;  // work areas: at most so many clusters or CTAs at once

int cal_setup(zola_psf* p, const zola_calib_data* cd, CalRun& run) {
    zola_ctx* ctx = p->ctx;
    if (!cd || !cd->dz || !cd->stacks) { ctx->err = "calibration: null data"; return ZOLA_E_ARG; }
    const int R = cd->R, nz = cd->nz, nb = cd->nbead, ns = cd->nslice;
    if (R < 4 || R % 2 || R > p->N || nz < 4 || nz > 231 || nb < 1 || ns < 1) {
        ctx->err = "calibration: need even R <= N, 4 <= nz <= 231, beads and slices >= 1";
        return ZOLA_E_ARG;
    }
    if (p->o.kz_reset) { ctx->err = "calibration: build the PSF with kz_reset = 0"; return ZOLA_E_ARG; }
    WindowTables* w = get_window(p, R, ctx->err);
    if (!w) return ZOLA_E_ARG;
    cudaSetDevice(ctx->device);
    if (int rc = cal_cuda(ctx, basis(p, nz))) return rc;
    CalView& V = run.V;
    V.D = p->D; V.a0 = p->a0; V.W = w->W; V.R = R; V.nb = nb; V.ns = ns; V.pb = 3 + ns + NPOLY;
    V.pupil = p->view.pupil; V.kx = p->view.kx; V.ky = p->view.ky; V.kzoil = p->view.kzoil; V.tw = p->view.tw;
    run.nz = nz;
    run.N = p->N;
    const size_t RR = (size_t)R * R, DD = (size_t)p->D * p->D, nbs = (size_t)nb * ns, WR = (size_t)R * w->W;
    run.per_cluster = cal_work_bytes(p->D, w->W, R);
    // The work buffers are carved from one grow-only area of the context, so that repeated
    // calls (an optimiser's forward / backward evaluations) allocate nothing.
    void** const q[] = {(void**)&run.d_par, (void**)&run.d_res, (void**)&run.d_phase, (void**)&run.d_slice,
                        (void**)&run.d_gphi, (void**)&run.d_gsum, (void**)&run.d_stacks, (void**)&run.d_const,
                        (void**)&run.scratch};
    const size_t n_par = run.head() + 2 * WR, n_res = 2 + nz + run.n_bead();
    const size_t bytes[] = {n_par * 8, n_res * 8, DD * 8, nbs * NOUT * 8, nbs * DD * 8, DD * 8, nbs * RR * 8,
                            (ns + (cd->photons ? nbs : 0)) * 8,
                            std::min<size_t>(CAL_CLUSTERS, nbs * 256) * run.per_cluster};
    cudaError_t e = carve(&ctx->calib_area, &ctx->calib_bytes, q, bytes, 9);
    cudaStream_t st = ctx->stream;
    if (e == cudaSuccess) e = copy_in(ctx, run.d_stacks, cd->stacks, nbs * RR * 8, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(run.d_const, cd->dz, (size_t)ns * 8, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && cd->photons)
        e = cudaMemcpyAsync(run.d_const + ns, cd->photons, nbs * 8, cudaMemcpyHostToDevice, st);
    if (int rc = cal_cuda(ctx, e)) return rc;
    run.par.resize(n_par);
    run.res.resize(n_res);
    V.dz = run.d_const;
    V.stacks = run.d_stacks;
    V.A0 = cd->photons ? run.d_const + ns : nullptr;
    V.GT = run.d_par + run.head();
    V.dGT = V.GT + WR;
    return ZOLA_OK;
}

// Coefficients, bead parameters and the blur tables at sigma; then the pupil phase.
int cal_upload(zola_psf* p, CalRun& run, const double* coef, double sigma, const double* bead) {
    zola_ctx* ctx = p->ctx;
    if (!(sigma > 0)) { ctx->err = "calibration: sigma must be positive"; return ZOLA_E_ARG; }
    const int R = run.V.R, W = run.V.W, DD = run.V.D * run.V.D;
    const size_t head = run.head();
    std::memcpy(run.par.data(), coef, run.nz * 8);
    const bool on_device = device_memory(bead);  // (as the driver's copies take it)
    if (!on_device) std::memcpy(run.par.data() + run.nz, bead, run.n_bead() * 8);
    size_t n = head;
    if (sigma != run.sigma) {
        std::vector<double> G, dG;
        blur_matrix(R, W, sigma, G, &dG);
        double* gt = run.par.data() + head;
        for (int i = 0; i < R; ++i)
            for (int k = 0; k < W; ++k) {
                gt[(size_t)k * R + i] = G[(size_t)i * W + k];
                gt[(size_t)(W + k) * R + i] = dG[(size_t)i * W + k];
            }
        run.sigma = sigma;
        n = run.par.size();
    }
    cudaError_t e = cudaMemcpyAsync(run.d_par, run.par.data(), n * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && on_device)
        e = cudaMemcpyAsync(run.d_par + run.nz, bead, run.n_bead() * 8, cudaMemcpyDeviceToDevice, ctx->stream);
    if (e == cudaSuccess) {
        k_cal_phase<<<(DD + 127) / 128, 128, 0, ctx->stream>>>(p->d_calZ, run.d_par, run.nz, DD, run.d_phase);
        ctx->launches++;
        e = cudaGetLastError();
    }
    return cal_cuda(ctx, e);
}

// Launch `kernel` with clusters of C CTAs for n items.
template <class KERNEL, class... ARGS>
cudaError_t cal_launch(zola_ctx* ctx, const CalRun& run, KERNEL kernel, int C, size_t n, ARGS... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(FL_THREADS);
    cfg.dynamicSmemBytes = cal_smem(run.N, run.V.D, run.V.W, run.V.R);
    cfg.stream = ctx->stream;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
    int at_once = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&at_once, kernel, &cfg);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3(C * (unsigned)std::min<size_t>(n, std::min(std::max(1, at_once), CAL_CLUSTERS)));
    ctx->launches++;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

int cal_eval(zola_psf* p, CalRun& run, const double* coef, double sigma, const double* bead, int mode, double* nll,
             double* gz, double* gsig, double* gb, double* model_dev, double* psi_dev) {
    zola_ctx* ctx = p->ctx;
    int rc = cal_upload(p, run, coef, sigma, bead);
    if (rc) return rc;
    const CalView& V = run.V;
    const int nbs = V.nb * V.ns, nz = mode ? run.nz : 0, DD = V.D * V.D;
    cudaStream_t st = ctx->stream;
    cudaError_t e = cudaSuccess;
    with_fft(run.N, [&](auto n) {
        e = cal_launch(ctx, run, k_cal_eval<decltype(n)::value>, f64_cluster(run.N, V.W), nbs, V,
                       (const double*)run.d_phase, (const double*)(run.d_par + run.nz), mode, run.K, run.scratch,
                       run.per_cluster, run.d_slice, run.d_gphi, model_dev, psi_dev);
    });
    if (e == cudaSuccess && mode) {
        k_cal_gsum<<<(DD + 31) / 32, 256, 0, st>>>(run.d_gphi, nbs, V.D, run.d_gsum);
        ctx->launches++;
    }
    if (e == cudaSuccess) {
        k_cal_finish<<<mode ? nz + V.nb + 1 : 1, 256, 0, st>>>(V, run.d_slice, run.d_gsum, p->d_calZ, nz, run.d_res);
        ctx->launches++;
        e = cudaGetLastError();
    }
    const size_t n = mode ? run.res.size() : 2;
    const bool on_device = mode && device_memory(gb);
    if (e == cudaSuccess) e = cudaMemcpyAsync(run.res.data(), run.d_res, n * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess && on_device)
        e = cudaMemcpyAsync(gb, run.d_res + 2 + nz, run.n_bead() * 8, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cal_cuda(ctx, e);
    *nll = run.res[0];
    if (!mode) return ZOLA_OK;
    if (gsig) *gsig = run.res[1];
    std::memcpy(gz, run.res.data() + 2, (size_t)nz * 8);
    if (!on_device) std::memcpy(gb, run.res.data() + 2 + nz, run.n_bead() * 8);
    return ZOLA_OK;
}

}  // namespace

extern "C" {

int zola_calib_forward(zola_psf* psf, const zola_calib_data* data, const double* zernike, double sigma,
                       const double* bead, double* nll, double* model) {
    if (!psf) return ZOLA_E_ARG;
    if (!zernike || !bead || !nll) { psf->ctx->err = "zola_calib_forward: null argument"; return ZOLA_E_ARG; }
    CalRun run;
    int rc = cal_setup(psf, data, run);
    if (rc) return rc;
    DevBuf<double> d_model;
    const size_t nm = (size_t)data->nbead * data->nslice * data->R * data->R;
    if (model && d_model.alloc(nm) != cudaSuccess) return ZOLA_E_CUDA;
    rc = cal_eval(psf, run, zernike, sigma, bead, 0, nll, nullptr, nullptr, nullptr, d_model.p, nullptr);
    if (rc) return rc;
    if (model && cudaMemcpy(model, d_model.p, nm * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return ZOLA_E_CUDA;
    return ZOLA_OK;
}

int zola_calib_backward(zola_psf* psf, const zola_calib_data* data, const double* zernike, double sigma,
                        const double* bead, double* nll, double* grad_zernike, double* grad_sigma, double* grad_bead) {
    if (!psf) return ZOLA_E_ARG;
    if (!zernike || !bead || !nll || !grad_zernike || !grad_bead) {
        psf->ctx->err = "zola_calib_backward: null argument";
        return ZOLA_E_ARG;
    }
    CalRun run;
    int rc = cal_setup(psf, data, run);
    if (rc) return rc;
    return cal_eval(psf, run, zernike, sigma, bead, 1, nll, grad_zernike, grad_sigma, grad_bead, nullptr, nullptr);
}

// LM over theta = (a_3..a_{nz-1}, [sigma], per bead x, y, z, a_bs, c_bk):
// gradient from the adjoint, Gauss-Newton matrix sum J J^T / mu from device
// tangents and per-slice Gram blocks, FP64 damped solve; a step is accepted
// when the NLL drops.  zernike / sigma / bead are updated in place.
int zola_calib_fit(zola_psf* psf, const zola_calib_data* data, double* zernike, double* sigma, double* bead,
                   int max_iter, int flags, double* nll_out, int* iters_out) {
    if (!psf) return ZOLA_E_ARG;
    zola_ctx* ctx = psf->ctx;
    if (!zernike || !sigma || !bead || !nll_out || max_iter < 0) {
        ctx->err = "zola_calib_fit: null argument or negative max_iter";
        return ZOLA_E_ARG;
    }
    CalRun run;
    int rc = cal_setup(psf, data, run);
    if (rc) return rc;
    const CalView& V = run.V;
    const int nz = data->nz, nzr = nz - 3, nb = data->nbead, ns = data->nslice, pb = V.pb;
    const size_t RR = (size_t)data->R * data->R, nbs = (size_t)nb * ns, DD = (size_t)V.D * V.D, WW = (size_t)V.W * V.W;
    const bool fit_sigma = (flags & ZOLA_CALIB_FIT_SIGMA) != 0;
    const int gsig = nzr;                         // theta index of sigma (when fitted)
    const int boff = nzr + (fit_sigma ? 1 : 0);   // first bead parameter
    const int npar = boff + nb * pb;
    const int nl = nzr + 5 + NPOLY;
    const size_t ne = (size_t)nl * (nl + 1) / 2;
    double *d_tan = nullptr, *d_model = nullptr, *d_psi = nullptr, *d_gram = nullptr, *d_H = nullptr, *d_A = nullptr,
           *d_g = nullptr;  // d_g: gradient, then the step and its flag
    void** const fq[] = {(void**)&d_tan, (void**)&d_model, (void**)&d_psi, (void**)&d_gram, (void**)&d_H, (void**)&d_A,
                         (void**)&d_g, (void**)&run.K.Q, (void**)&run.K.E, (void**)&run.K.T, (void**)&run.K.Ts,
                         (void**)&run.K.S};
    const size_t n2 = (size_t)npar * npar;
    const size_t bead_rows = (size_t)pb + boff + 1;
    const size_t fb[] = {(nzr + 4) * nbs * RR * 8, nbs * RR * 8, nbs * RR * 8, nbs * ne * 8, n2 * 8,
                         (nb * bead_rows * bead_rows + (size_t)(boff + 1) * boff) * 8, (2 * (size_t)npar + 1) * 8, nbs * DD * 16, nbs * WW * 16, nbs * RR * 8,
                         nbs * RR * 8, nbs * 8};
    if (carve(&ctx->calib_fit_area, &ctx->calib_fit_bytes, fq, fb, 12) != cudaSuccess) {
        ctx->err = "zola_calib_fit: device memory";
        return ZOLA_E_CUDA;
    }
    const size_t gn_smem = ((size_t)GN_CHUNK * (gn_stride(nl) + 1) + 16 * FL_THREADS / 2) * 8;
    if (cudaFuncSetAttribute(k_cal_gn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gn_smem) != cudaSuccess ||
        cudaFuncSetAttribute(k_cal_bead, cudaFuncAttributeMaxDynamicSharedMemorySize, CH_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(k_cal_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, CH_SMEM) != cudaSuccess) {
        ctx->err = "zola_calib_fit: shared memory";
        return ZOLA_E_CUDA;
    }
    std::vector<double> th(npar), g(npar), gz(nz), gb((size_t)nb * pb);
    std::vector<double> A0;
    if (data->photons) A0.assign(data->photons, data->photons + nbs);
    std::vector<double> zc(zernike, zernike + nz), bd(bead, bead + (size_t)nb * pb);
    double sg = *sigma;
    auto pack = [&](std::vector<double>& t) {
        for (int i = 0; i < nzr; ++i) t[i] = zernike[i + 3];
        if (fit_sigma) t[gsig] = *sigma;
        for (int k = 0; k < nb * pb; ++k) t[boff + k] = bead[k];
    };
    auto unpack = [&](const std::vector<double>& t) {
        for (int i = 0; i < nzr; ++i) zc[i + 3] = t[i];
        if (fit_sigma) sg = t[gsig];
        for (int k = 0; k < nb * pb; ++k) bd[k] = t[boff + k];
    };
    auto evaluate = [&](const std::vector<double>& t, double* f, std::vector<double>& grad) -> int {
        unpack(t);
        double gs = 0;
        int r = cal_eval(psf, run, zc.data(), sg, bd.data(), 1, f, gz.data(), &gs, gb.data(), d_model, d_psi);
        if (r) return r;
        for (int i = 0; i < nzr; ++i) grad[i] = gz[i + 3];
        if (fit_sigma) grad[gsig] = gs;
        for (int k = 0; k < nb * pb; ++k) grad[boff + k] = gb[k];
        return 0;
    };
    // Gauss-Newton matrix at the point of the last evaluation
    auto matrix = [&]() -> int {
        cudaStream_t st = ctx->stream;
        cudaError_t e = cudaSuccess;
        with_fft(run.N, [&](auto n) {
            e = cal_launch(ctx, run, k_cal_tangent<decltype(n)::value>, 1, (size_t)(nzr + 4) * nbs, V, run.K,
                           (const double*)(run.d_par + run.nz), (const double*)psf->d_calZ, nzr, run.scratch,
                           run.per_cluster, d_tan);
        });
        if (e == cudaSuccess) {
            k_cal_gn<<<(unsigned)std::min<size_t>(nbs, 4096), FL_THREADS, gn_smem, st>>>(V, nzr, d_tan, d_model, d_psi,
                                                                                         d_gram);
            const dim3 grid((npar + 31) / 32, (npar + 7) / 8);
            k_cal_hess<<<grid, dim3(32, 8), 0, st>>>(V, nzr, fit_sigma, npar, d_gram, d_H);
            ctx->launches += 2;
            e = cudaGetLastError();
        }
        return cal_cuda(ctx, e);
    };
    auto solve = [&](const std::vector<double>& grad, double lambda, std::vector<double>& step, bool* ok) -> int {
        cudaStream_t st = ctx->stream;
        int flag = 0;
        double *x = d_g + npar, *S = d_A + nb * bead_rows * bead_rows;
        int* flags = (int*)(d_g + 2 * npar);
        cudaError_t e = cudaMemcpyAsync(d_g, grad.data(), (size_t)npar * 8, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(flags, 0xff, sizeof(int), st);
        if (e == cudaSuccess) {
            k_cal_bead<<<nb, CH_THREADS, CH_SMEM, st>>>(d_H, d_g, npar, boff, pb, lambda, d_A, flags);
            k_cal_shared<<<1, CH_THREADS, CH_SMEM, st>>>(d_H, d_g, npar, boff, pb, nb, lambda, d_A, S, x, flags);
            k_cal_back<<<nb, CH_THREADS, CH_B * 8, st>>>(boff, pb, d_A, x, flags);
            ctx->launches += 3;
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(step.data(), d_g + npar, (size_t)npar * 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, d_g + 2 * npar, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        *ok = flag != 0;
        return cal_cuda(ctx, e);
    };
    auto constrain = [&](std::vector<double>& t) {
        if (fit_sigma) t[gsig] = std::max(t[gsig], 0.05);
        for (int b = 0; b < nb; ++b)
            for (int s = 0; s < ns; ++s) {
                const double a0 = A0.empty() ? 0.0 : A0[(size_t)b * ns + s];
                double& a = t[boff + b * pb + 3 + s];
                a = std::max(a, 1.0 - a0);  // total photons >= 1
            }
    };
    pack(th);
    double nll = 0, lambda = 1e-3;
    int it = 0;
    std::vector<double> step(npar), g2(npar);
    rc = evaluate(th, &nll, g);
    if (rc) return rc;
    bool stale = true;  // the matrix is formed when a step is solved for
    for (it = 0; it < max_iter; ++it) {
        bool ok = false;
        if (stale && (rc = matrix())) return rc;
        stale = false;
        if ((rc = solve(g, lambda, step, &ok))) return rc;
        if (!ok) {
            lambda *= 10;
            if (lambda > 1e10) break;
            continue;
        }
        std::vector<double> t2(th);
        for (int i = 0; i < npar; ++i) t2[i] += step[i];
        constrain(t2);
        double nll2;
        rc = evaluate(t2, &nll2, g2);
        if (rc) return rc;
        if (nll2 <= nll) {
            const double dec = nll - nll2;
            th = t2;
            nll = nll2;
            g.swap(g2);
            stale = true;
            lambda = std::max(lambda * 0.1, 1e-9);
            if (dec < 1e-9 * std::max(1.0, std::fabs(nll))) { ++it; break; }
        } else {
            lambda *= 10;
            if (lambda > 1e10) break;
        }
    }
    unpack(th);
    std::memcpy(zernike, zc.data(), (size_t)nz * 8);
    std::memcpy(bead, bd.data(), bd.size() * 8);
    *sigma = sg;
    *nll_out = nll;
    if (iters_out) *iters_out = it;
    return ZOLA_OK;
}

}  // extern "C"
