// FP64 Fourier transforms inside a CTA: complex arithmetic, small DFTs, and the
// transform of LINES lines of N = 4 .. 1024 points by 256 threads; clusters.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

namespace zola {

__device__ inline double2 c_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ inline double2 c_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ inline double2 c_mul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
// a times exp(SIGN i pi / 2)
template <int SIGN>
__device__ inline double2 c_rot(double2 a) { return SIGN > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x); }

template <int SIGN>
__device__ inline void dft3(double2& a, double2& b, double2& c) {
    const double h = 0.86602540378443864676;  // sin(2 pi / 3)
    const double2 s = c_add(b, c), d = c_rot<SIGN>(make_double2(h * (b.x - c.x), h * (b.y - c.y)));
    const double2 m = make_double2(fma(-0.5, s.x, a.x), fma(-0.5, s.y, a.y));
    a = c_add(a, s);
    b = c_add(m, d);
    c = c_sub(m, d);
}

template <int SIGN>
__device__ inline void dft4(double2& a, double2& b, double2& c, double2& d) {
    const double2 s0 = c_add(a, c), s1 = c_sub(a, c), s2 = c_add(b, d), s3 = c_rot<SIGN>(c_sub(b, d));
    a = c_add(s0, s2);
    b = c_add(s1, s3);
    c = c_sub(s0, s2);
    d = c_sub(s1, s3);
}

template <int SIGN, int R>
__device__ inline void dft(double2 (&x)[R]) {
    if constexpr (R == 4) {
        dft4<SIGN>(x[0], x[1], x[2], x[3]);
    } else if constexpr (R == 5) {
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;  // cos(2 pi k / 5)
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;   // sin(2 pi k / 5)
        const double2 p = c_add(x[1], x[4]), q = c_add(x[2], x[3]), u = c_sub(x[1], x[4]), v = c_sub(x[2], x[3]);
        const double2 e = make_double2(fma(c1, p.x, fma(c2, q.x, x[0].x)), fma(c1, p.y, fma(c2, q.y, x[0].y)));
        const double2 f = make_double2(fma(c2, p.x, fma(c1, q.x, x[0].x)), fma(c2, p.y, fma(c1, q.y, x[0].y)));
        const double2 g = c_rot<SIGN>(make_double2(fma(s1, u.x, s2 * v.x), fma(s1, u.y, s2 * v.y)));
        const double2 h = c_rot<SIGN>(make_double2(fma(s2, u.x, -s1 * v.x), fma(s2, u.y, -s1 * v.y)));
        x[0] = c_add(x[0], c_add(p, q));
        x[1] = c_add(e, g);
        x[4] = c_sub(e, g);
        x[2] = c_add(f, h);
        x[3] = c_sub(f, h);
    } else if constexpr (R == 6) {  // 2 x 3, prime factors: inputs (3a + 2b) mod 6, outputs (3a + 4b) mod 6
        double2 a[3] = {x[0], x[2], x[4]}, b[3] = {x[3], x[5], x[1]};
        dft3<SIGN>(a[0], a[1], a[2]);
        dft3<SIGN>(b[0], b[1], b[2]);
        x[0] = c_add(a[0], b[0]);
        x[3] = c_sub(a[0], b[0]);
        x[4] = c_add(a[1], b[1]);
        x[1] = c_sub(a[1], b[1]);
        x[2] = c_add(a[2], b[2]);
        x[5] = c_sub(a[2], b[2]);
    } else if constexpr (R == 8) {
        const double h = 0.70710678118654752440;
        double2 a[4] = {x[0], x[2], x[4], x[6]}, b[4] = {x[1], x[3], x[5], x[7]};
        dft4<SIGN>(a[0], a[1], a[2], a[3]);
        dft4<SIGN>(b[0], b[1], b[2], b[3]);
        const double2 r1 = c_rot<SIGN>(b[1]), r3 = c_rot<SIGN>(b[3]);
        b[1] = make_double2(h * (b[1].x + r1.x), h * (b[1].y + r1.y));
        b[2] = c_rot<SIGN>(b[2]);
        b[3] = make_double2(h * (r3.x - b[3].x), h * (r3.y - b[3].y));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q] = c_add(a[q], b[q]);
            x[q + 4] = c_sub(a[q], b[q]);
        }
    }
}

// N-point lines, N a power of two: fl_lines(N) lines at once, 256 threads, a 32 KB
// buffer [point][line].  A thread owns one radix-8 or two radix-4 butterflies a
// pass (one at N = 4, where a line has no more and there are only as many lines as
// threads), its operands stay in registers over the barrier, and it ends with eight
// outputs (four at N = 4), always the same (point, line) for a given thread, so that results of
// several transforms can be combined in registers.  The lane index runs over the
// lines first: shared-memory accesses are conflict-free and few twiddles differ.
constexpr int FL_THREADS = 256, FL_OUT = 8;
__host__ __device__ constexpr int fl_lines(int N) { return N < 8 ? FL_THREADS : 2048 / N; }
template <int N_>
struct FftLines {
    static constexpr int N = N_, LINES = fl_lines(N_);
    static constexpr int R0 = N == 4 || N == 16 ? 4 : 8, R1 = N <= 8 ? 1 : (N <= 32 || N == 128 ? 4 : 8),
                         R2 = N <= 64 ? 1 : (N == 512 ? 8 : 4), R3 = N == 1024 ? 4 : 1;
    static_assert(R0 * R1 * R2 * R3 == N, "4 .. 1024 points");
    static_assert(LINES <= FL_THREADS && LINES * N <= FL_OUT * FL_THREADS, "a line a thread");
};
constexpr size_t FL_SMEM = 2048 * sizeof(double2);

template <class F, int SIGN, int R, int NS, class LD, class ST>
__device__ __forceinline__ void fl_pass(double2* sm, const double2* tw, const LD& ld, const ST& st) {
    constexpr int B = F::LINES * F::N / (FL_THREADS * R);  // butterflies a thread
    constexpr bool first = NS == 1, last = NS * R == F::N;
    constexpr unsigned nb = F::N / R, JS = FL_THREADS / F::LINES;
    const unsigned line = threadIdx.x % F::LINES, j0 = threadIdx.x / F::LINES;
    double2 x[B][R];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const unsigned j = j0 + b * JS, k = first ? 0 : j % NS;
#pragma unroll
        for (unsigned q = 0; q < R; ++q) x[b][q] = first ? ld(j + q * nb, line) : sm[(j + q * nb) * F::LINES + line];
        if (!first) {
#pragma unroll
            for (unsigned q = 1; q < R; ++q) {
                double2 w = __ldg(tw + q * k * (nb / NS));
                if (SIGN > 0) w.y = -w.y;
                x[b][q] = c_mul(x[b][q], w);
            }
        }
        dft<SIGN, R>(x[b]);
    }
    if (!first && !last) __syncthreads();  // every operand is in registers before the buffer is overwritten
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const unsigned j = j0 + b * JS, k = first ? 0 : j % NS, o = (j - k) * R + k;
#pragma unroll
        for (unsigned q = 0; q < R; ++q) {
            if (last) st(o + q * NS, line, b * R + (int)q, x[b][q]);
            else sm[(o + q * NS) * F::LINES + line] = x[b][q];
        }
    }
    if (!last) __syncthreads();
}

// The transform exp(SIGN 2 pi i j k / N) of the CTA's lines: ld(point, line) gives
// the input, st(point, line, slot, value) takes the output (slot 0 .. 7 of this
// thread).  tw[k] = exp(-2 pi i k / N).  The buffer is free again after the next
// barrier; a caller that starts another transform has one in between.
template <class F, int SIGN, class LD, class ST>
__device__ __forceinline__ void fl_transform(double2* sm, const double2* tw, const LD& ld, const ST& st) {
    fl_pass<F, SIGN, F::R0, 1>(sm, tw, ld, st);
    if constexpr (F::R1 > 1) fl_pass<F, SIGN, F::R1, F::R0>(sm, tw, ld, st);
    if constexpr (F::R2 > 1) fl_pass<F, SIGN, F::R2, F::R0 * F::R1>(sm, tw, ld, st);
    if constexpr (F::R3 > 1) fl_pass<F, SIGN, F::R3, F::R0 * F::R1 * F::R2>(sm, tw, ld, st);
}

constexpr int FL_WARPS = FL_THREADS / 32;

// The CTAs of a cluster share one ROI, model or bead slice: each takes its part of the pupil
// rows, of the window columns and of the pixel rows, and they meet at cluster
// barriers.  An evaluation then takes a fraction of the time, which is what one ROI,
// a few of them, or the last slow fits of a batch wait for.
struct Cluster {
    unsigned rank, size;
    __device__ Cluster() {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    }
    __device__ void sync() const {
        if (size == 1) __syncthreads();
        else asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    }
    // p (in this CTA's shared memory) as CTA r of the cluster has it
    template <class T>
    __device__ T read(const T* p, unsigned r) const { return *cooperative_groups::this_cluster().map_shared_rank((T*)p, r); }
    __device__ unsigned id() const { return blockIdx.x / size; }
    __device__ unsigned count() const { return gridDim.x / size; }
    // this CTA's part of the row pairs of an R x R map
    __device__ int row0(int R) const { return (int)(R / 2 * rank / size) * 2; }
    __device__ int row1(int R) const { return (int)(R / 2 * (rank + 1) / size) * 2; }
};
// CTAs a cluster, by the window's columns (LINES at a time); never by the number of
// ROIs, so that a result does not depend on its batch.
__host__ __device__ inline int f64_cluster(int N, int W) {
    const int t = W / fl_lines(N);
    return t >= 4 ? 4 : (t >= 2 ? 2 : 1);
}

// Sum of NV doubles per thread over the cluster; every thread gets it.  red: 9 NV
// doubles, part: NV doubles of shared memory not used by the previous call.
template <int NV>
__device__ inline void cluster_sum(const Cluster& cl, double (&v)[NV], double* red, double* part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        v[k] = x;
    }
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) red[warp * NV + k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < FL_WARPS; ++w) s += red[w * NV + threadIdx.x];
        part[threadIdx.x] = s;
    }
    cl.sync();
    if (threadIdx.x < NV) {
        double s = part[threadIdx.x];
        if (cl.size > 1) {
            s = 0.0;
            for (unsigned r = 0; r < cl.size; ++r) s += cl.read(part + threadIdx.x, r);
        }
        red[FL_WARPS * NV + threadIdx.x] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = red[FL_WARPS * NV + k];
}

// J[i'][c0 + c] = sum_i G[i'][i] X[i][c] for a shared tile X (W x L, L the row stride)
// of `cols` columns: two rows i' by two columns a thread, two 16-byte loads for four
// FMAs.  GT = the transposed blur matrix (W x R).  J has W columns.
__device__ __forceinline__ void blur_tile(const double* GT, const double* X, int R, int W, int L, int cols, double* J) {
    const int hc = cols / 2;
    for (int t = threadIdx.x; t < (R / 2) * hc; t += FL_THREADS) {
        const int rp = t / hc, c = t - rp * hc;
        const double *g = GT + 2 * rp, *xi = X + 2 * c;
        double s00 = 0, s01 = 0, s10 = 0, s11 = 0;
#pragma unroll 4
        for (int i = 0; i < W; ++i) {
            const double2 gv = *(const double2*)(g + (size_t)i * R), xv = *(const double2*)(xi + i * L);
            s00 = fma(gv.x, xv.x, s00);
            s01 = fma(gv.x, xv.y, s01);
            s10 = fma(gv.y, xv.x, s10);
            s11 = fma(gv.y, xv.y, s11);
        }
        *(double2*)(J + (size_t)(2 * rp) * W + 2 * c) = make_double2(s00, s01);
        *(double2*)(J + (size_t)(2 * rp + 1) * W + 2 * c) = make_double2(s10, s11);
    }
}

// fn(integral constant N): the transforms of an N-point pupil grid.
template <class FN>
inline void with_fft(int N, const FN& fn) {
    switch (N) {
        case 4: fn(std::integral_constant<int, 4>()); break;
        case 8: fn(std::integral_constant<int, 8>()); break;
        case 16: fn(std::integral_constant<int, 16>()); break;
        case 32: fn(std::integral_constant<int, 32>()); break;
        case 64: fn(std::integral_constant<int, 64>()); break;
        case 128: fn(std::integral_constant<int, 128>()); break;
        case 256: fn(std::integral_constant<int, 256>()); break;
        case 512: fn(std::integral_constant<int, 512>()); break;
        case 1024: fn(std::integral_constant<int, 1024>()); break;
    }
}

}  // namespace zola
