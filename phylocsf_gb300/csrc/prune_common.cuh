// Device helpers shared by the pruning and gradient kernels.
#pragma once
#include <cuda_runtime.h>

#include "pcsf_internal.h"

namespace pcsf {

// Pairs of floats (one 64-bit register pair), elementwise round-to-nearest: two lanes' work in one
// issue slot at the scalar rate (measured 127 lanes per clock and SM either way).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float x, float y) { f2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y)); return d; }
__device__ __forceinline__ void upk(f2 a, float &x, float &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { f2 d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 neg2(f2 a) { return a ^ 0x8000000080000000ull; }

template <typename T> struct Vec4;
template <> struct Vec4<float> {
    static __device__ inline void load(const float *p, float v[4])
    {
        float4 x = *reinterpret_cast<const float4 *>(p);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
};
template <> struct Vec4<double> {
    static __device__ inline void load(const double *p, double v[4])
    {
        double2 x = *reinterpret_cast<const double2 *>(p);
        double2 y = *reinterpret_cast<const double2 *>(p + 2);
        v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
    }
};

template <typename T> struct AtomMax;
template <> struct AtomMax<float> {
    typedef int U;
    static __device__ inline void upd(U *p, float v) { atomicMax(p, __float_as_int(v)); }
    static __device__ inline float get(const U *p) { return __int_as_float(*p); }
};
template <> struct AtomMax<double> {
    typedef unsigned long long U;
    static __device__ inline void upd(U *p, double v) { atomicMax(p, (unsigned long long)__double_as_longlong(v)); }
    static __device__ inline double get(const U *p) { return __longlong_as_double((long long)*p); }
};

template <typename T, int CPT> struct ColLoad;
template <typename T> struct ColLoad<T, 1> {
    static __device__ inline void load(const T *p, T v[1]) { v[0] = p[0]; }
};
template <> struct ColLoad<float, 4> {
    static __device__ inline void load(const float *p, float v[4]) { Vec4<float>::load(p, v); }
};
template <> struct ColLoad<float, 2> {
    static __device__ inline void load(const float *p, float v[2])
    {
        float2 x = *reinterpret_cast<const float2 *>(p);
        v[0] = x.x; v[1] = x.y;
    }
};
template <> struct ColLoad<double, 2> {
    static __device__ inline void load(const double *p, double v[2])
    {
        double2 x = *reinterpret_cast<const double2 *>(p);
        v[0] = x.x; v[1] = x.y;
    }
};
template <> struct ColLoad<double, 4> {
    static __device__ inline void load(const double *p, double v[4]) { Vec4<double>::load(p, v); }
};

template <typename T, int CPT> struct ColStore;
template <> struct ColStore<float, 4> {
    static __device__ inline void store(float *p, const float v[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};
template <typename T> struct ColStore<T, 1> {
    static __device__ inline void store(T *p, const T v[1]) { *p = v[0]; }
};
template <> struct ColStore<float, 2> {
    static __device__ inline void store(float *p, const float v[2]) { *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]); }
};
template <> struct ColStore<double, 2> {
    static __device__ inline void store(double *p, const double v[2]) { *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]); }
};
template <> struct ColStore<double, 4> {
    static __device__ inline void store(double *p, const double v[4])
    {
        *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2 *>(p + 2) = make_double2(v[2], v[3]);
    }
};

// P(t) status keys: first error in (branch, row) order wins
__device__ __forceinline__ void status_min(int32_t *key, int branch, int row, int code)
{
    atomicMin(key, ((branch * K + row) << 4) | code);
}

// Tensor-core B operand of E (rows a, K = j): TF32 hi / lo parts in the K-major
// core-matrix layout of the tensor-core kernel (tc_kernels.cu), 16 KB each:
// element (a, j) at float offset (j/4)*256 + a*4 + j%4 of its part.
__device__ __forceinline__ void bop_store(float *dst, int a, int q, float4 x)
{
    // hi rounded to the nearest TF32 value (as tf32_hi in tc_common.cuh), lo = x - hi exact
    const float4 h = make_float4(__uint_as_float((__float_as_uint(x.x) + 0x1000u) & 0xFFFFE000u),
                                 __uint_as_float((__float_as_uint(x.y) + 0x1000u) & 0xFFFFE000u),
                                 __uint_as_float((__float_as_uint(x.z) + 0x1000u) & 0xFFFFE000u),
                                 __uint_as_float((__float_as_uint(x.w) + 0x1000u) & 0xFFFFE000u));
    const float4 l = make_float4(x.x - h.x, x.y - h.y, x.z - h.z, x.w - h.w);
    *reinterpret_cast<float4 *>(dst + q * 256 + a * 4) = h;
    *reinterpret_cast<float4 *>(dst + K2 + q * 256 + a * 4) = l;
}

// Row sum of the raw P(t) minus one, through the eigensystem: isq_i sum_m U_im
// expm1(lam_m t) w_m, where only the stationary direction(s) have w_m != 0;
// ex[m] = expm1(lam_m t) must be valid for those m.
__device__ __forceinline__ double rowsum_minus_one(const DevModels &m, int md, int i, const double *ex)
{
    const double *U = m.U + (size_t)md * K2 + (size_t)i * K;
    const double *w = m.wrow + md * K;
    const int16_t *wl = m.wlist + md * WLIST;
    double rs = 0.0;
    if (wl[0] == -2) {
        for (int mm = 0; mm < K; mm++)
            if (w[mm] != 0.0) rs += U[mm] * ex[mm] * w[mm];
    } else {
        for (int k = 0; k < WLIST && wl[k] >= 0; k++) rs += U[wl[k]] * ex[wl[k]] * w[wl[k]];
    }
    return rs * m.isq[md * K + i];
}

// Grid point nearest to t >= grid_t[0].  FP32 places t to about a thousandth of a step, and the
// comparison with the next point makes the choice: from a point off by one, where t is that close
// to a grid point, it is the same one.  (The FP64 logarithm and divisions were 4,000 clocks.)
__device__ __forceinline__ int grid_point(const DevModels &m, double t)
{
    int g = (int)floorf(logf((float)t / (float)m.grid_t[0]) / (float)m.grid_lr);
    g = max(0, min(g, m.grid_n - 1));
    if (g + 1 < m.grid_n && (m.grid_t[g + 1] - t) < (t - m.grid_t[g])) g++;
    return g;
}

// Per-column dithering of the leaf partials (SIMT FP32 pruning): each leaf partial
// of column col is scaled by the exact factor c = 1 + k/256, k = dither_k(col, leaf),
// and sum_leaves log c is subtracted from the column's log-likelihood.  The values
// are mathematically unchanged; the FP32 rounding errors of columns that share
// sub-patterns (the same states below a node) stop being identical, so they no
// longer add up linearly over thousands of columns.
__device__ __forceinline__ int dither_k(int64_t col, int leaf)
{
    uint32_t h = (uint32_t)col * 0x9E3779B1u + (uint32_t)((uint64_t)col >> 32) * 0x7FEB352Du + (uint32_t)leaf * 0x85EBCA77u;
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    h *= 0x297A2D39u;
    h ^= h >> 15;
    return (int)(h & 255u);
}

// Where k_prune_tc's leaf rows keep state a (its own inverse): within each 32 states, the four
// pairs a thread of the row fragment holds are consecutive, 32 bytes.
__device__ __forceinline__ int leaf_pos(int a) { return (a & 33) | ((a >> 2) & 6) | ((a << 2) & 24); }

// exp_of(x): the e of frexp (x = m 2^e, m in [0.5, 1)) read from the exponent
// field for normal x; frexp itself for zero, subnormals and non-finite x.
__device__ __forceinline__ int exp_of(float x)
{
    const int b = (__float_as_int(x) >> 23) & 0xff;
    if (b != 0 && b != 0xff) return b - 126;
    int e;
    frexpf(x, &e);
    return e;
}
__device__ __forceinline__ int exp_of(double x)
{
    const int b = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
    if (b != 0 && b != 0x7ff) return b - 1022;
    int e;
    frexp(x, &e);
    return e;
}
// 2^e, |e| <= 126 (float) / 1022 (double)
template <typename T> __device__ __forceinline__ T pow2(int e);
template <> __device__ __forceinline__ float pow2<float>(int e) { return __int_as_float((e + 127) << 23); }
template <> __device__ __forceinline__ double pow2<double>(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// scale2(x, e) = x * 2^e as two multiplications by exact powers of two (e split
// in halves of equal sign, so the intermediate lies between x and the result):
// exact, like ldexp, whenever x and the result are normal or zero; |e| <= 252
// (float) / 2044 (double), far beyond the per-node rescales.
template <typename T>
__device__ __forceinline__ T scale2(T x, int e)
{
    const int e1 = e >> 1, e2 = e - e1;
    return x * pow2<T>(e1) * pow2<T>(e2);
}

// out[i][cc] = sum_j M[j][a0+i] * X[j][c0+cc] for a 64 x TC shared-memory tile
// X ([K][TC]) and a 64 x 64 matrix M ([K][K], row j contiguous).
// COMP selects the summation: 0 plain FP32 (products smaller than half an ulp of
// the running sum are lost, a downward bias), 1 Kahan on every term, 2 blocked:
// eight products summed plainly, then each block folded into the running sum
// with Kahan's correction (about a ninth of the plain bias at 1.5 operations per
// product instead of 5).
// CPT: columns per thread (TC / 16 with 256 threads of 4 states each).
// FP32 with two or four columns per thread works on pairs of columns (contract_pairs).
template <typename T, int TC, int COMP, int CPT = TC / 16, int UNROLL = 1>
__device__ inline void contract_scalar(const T *M, const T *X, int a0, int c0, T out[4][CPT])
{
    T comp[4][CPT];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int cc = 0; cc < CPT; cc++) {
            out[i][cc] = (T)0;
            comp[i][cc] = (T)0;
        }
    if (COMP == 2) {
        // a block's sum starts from its first product (0 + p rounds as p does), and the
        // first block is the running sum itself (its fold into zeros is exact, with a
        // zero correction): the same values as zero-initialised sums and folds, with
        // fewer instructions in this issue-bound loop
        auto block = [&](int jb, T g[4][CPT]) {
#pragma unroll
            for (int j = jb; j < jb + 8; j++) {
                T e[4], x[CPT];
                Vec4<T>::load(M + j * K + a0, e);
                ColLoad<T, CPT>::load(X + j * TC + c0, x);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) g[i][cc] = (j == jb) ? e[i] * x[cc] : fma(e[i], x[cc], g[i][cc]);
            }
        };
        block(0, out);
#pragma unroll UNROLL
        for (int jb = 8; jb < K; jb += 8) {
            T g[4][CPT];
            block(jb, g);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    T y = g[i][cc] - comp[i][cc];
                    T t = out[i][cc] + y;
                    comp[i][cc] = (t - out[i][cc]) - y;
                    out[i][cc] = t;
                }
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < K; j++) {
            T e[4], x[CPT];
            Vec4<T>::load(M + j * K + a0, e);
            ColLoad<T, CPT>::load(X + j * TC + c0, x);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    if (COMP == 1) {
                        // compensated summation: the rounding error of each addition is
                        // carried in comp, so small terms are not lost against a large sum
                        T y = e[i] * x[cc] - comp[i][cc];
                        T t = out[i][cc] + y;
                        comp[i][cc] = (t - out[i][cc]) - y;
                        out[i][cc] = t;
                    } else {
                        out[i][cc] += e[i] * x[cc];
                    }
                }
        }
    }
    if (COMP) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) out[i][cc] -= comp[i][cc];
    }
}

// The same sums on pairs of columns: bit for bit the scalar values (each lane rounds as the scalar
// operation), with half of the issue slots for products and corrections.  The loop is issue-bound:
// 208 instructions per 8 products of a 4 x 4 block before, 64 + 32 paired ones, 16 loads and the
// duplication of E's entries now.  The correction is kept negated (a + (-c) rounds as a - c).
// Measured with the staged leaf rows, blocked compensation, 58 leaves, 141,741 columns: 3.12 ->
// 2.68 ms; what bounds it now is the mix of FP32 issue, load latency and three barriers a node.
// entry(j, e): E's four entries of step j.
// UNROLL: blocks of the compensated sum in a row (7: all of them).  Rolled, each block begins with
// its loads' latency (k_prune 2.94 ms against 2.68 with 7); unrolled, a kernel with many contractions
// outgrows the instruction cache (k_grad with 1 / 3 / 7: 58 leaves 6.43 / 6.19 / 6.47 ms, 100 leaves
// with rate parameters 12.6 / 12.2 / 15.7 ms).
template <int TC, int COMP, int CPT, int UNROLL, typename Entry>
__device__ inline void contract_pairs(Entry entry, const float *X, int c0, float out[4][CPT])
{
    constexpr int NP = CPT / 2;
    f2 s[4][NP], nc[4][NP];
    auto load_x = [&](int j, f2 x[NP]) {
        float v[CPT];
        ColLoad<float, CPT>::load(X + j * TC + c0, v);
#pragma unroll
        for (int k = 0; k < NP; k++) x[k] = pk(v[2 * k], v[2 * k + 1]);
    };
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int k = 0; k < NP; k++) s[i][k] = nc[i][k] = 0ull;
    if (COMP == 2) {
        auto block = [&](int jb, f2 g[4][NP]) {
#pragma unroll
            for (int j = jb; j < jb + 8; j++) {
                float e[4];
                f2 x[NP];
                entry(j, e);
                load_x(j, x);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const f2 ee = pk(e[i], e[i]);
#pragma unroll
                    for (int k = 0; k < NP; k++) g[i][k] = (j == jb) ? mul2(ee, x[k]) : fma2(ee, x[k], g[i][k]);
                }
            }
        };
        block(0, s);
#pragma unroll UNROLL
        for (int jb = 8; jb < K; jb += 8) {
            f2 g[4][NP];
            block(jb, g);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int k = 0; k < NP; k++) {
                    const f2 y = add2(g[i][k], nc[i][k]);
                    const f2 t = add2(s[i][k], y);
                    nc[i][k] = sub2(y, sub2(t, s[i][k]));
                    s[i][k] = t;
                }
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < K; j++) {
            float e[4];
            f2 x[NP];
            entry(j, e);
            load_x(j, x);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const f2 ee = pk(e[i], e[i]);
#pragma unroll
                for (int k = 0; k < NP; k++) {
                    if (COMP == 1) {
                        const f2 y = fma2(ee, x[k], nc[i][k]);
                        const f2 t = add2(s[i][k], y);
                        nc[i][k] = sub2(y, sub2(t, s[i][k]));
                        s[i][k] = t;
                    } else {
                        s[i][k] = fma2(ee, x[k], s[i][k]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int k = 0; k < NP; k++) upk(COMP ? add2(s[i][k], nc[i][k]) : s[i][k], out[i][2 * k], out[i][2 * k + 1]);
}

template <typename T, int TC, int COMP, int CPT = TC / 16, int UNROLL = 1>
__device__ inline void contract(const T *M, const T *X, int a0, int c0, T out[4][CPT])
{
    if constexpr (sizeof(T) == 4 && CPT % 2 == 0)
        contract_pairs<TC, COMP, CPT, UNROLL>([&](int j, float e[4]) { Vec4<float>::load(M + j * K + a0, e); }, X, c0, out);
    else
        contract_scalar<T, TC, COMP, CPT, UNROLL>(M, X, a0, c0, out);
}

// out[i][cc] = sum_j N[a0+i][j] * X[j][c0+cc] with row a of N at N + a * LDN: contract() of the
// transposed matrix (the same products in the same order, so the same values), for the outside
// pass, which multiplies by E^T as it is stored.  Four consecutive j of a row come in one load;
// LDN = K + 4 keeps the two row groups of a warp on different banks.
constexpr int LDN = K + 4;
template <typename T, int TC, int COMP, int UNROLL = 1>
__device__ inline void contract_rows(const T *N, const T *X, int a0, int c0, T out[4][TC / 16])
{
    constexpr int CPT = TC / 16;
    if constexpr (sizeof(T) == 4 && CPT % 2 == 0) {
        float r[4][4];       // four steps of the thread's four rows
        contract_pairs<TC, COMP, CPT, UNROLL>(
            [&](int j, float e[4]) {
                if (j % 4 == 0) {
#pragma unroll
                    for (int i = 0; i < 4; i++) Vec4<float>::load(N + (a0 + i) * LDN + j, r[i]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) e[i] = r[i][j % 4];
            },
            X, c0, out);
        return;
    }
    T comp[4][CPT];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int cc = 0; cc < CPT; cc++) {
            out[i][cc] = (T)0;
            comp[i][cc] = (T)0;
        }
    // sum (or, first = true, start) of J products from j0
    auto products = [&](int j0, T g[4][CPT], bool first) {
        T e[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++) Vec4<T>::load(N + (a0 + i) * LDN + j0, e[i]);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            T x[CPT];
            ColLoad<T, CPT>::load(X + (j0 + j) * TC + c0, x);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    if (COMP == 1) {
                        const T y = e[i][j] * x[cc] - comp[i][cc];
                        const T t = g[i][cc] + y;
                        comp[i][cc] = (t - g[i][cc]) - y;
                        g[i][cc] = t;
                    } else if (COMP == 2) {
                        g[i][cc] = (first && j == 0) ? e[i][j] * x[cc] : fma(e[i][j], x[cc], g[i][cc]);
                    } else {
                        g[i][cc] += e[i][j] * x[cc];
                    }
                }
        }
    };
    if (COMP == 2) {
        products(0, out, true);
        products(4, out, false);
#pragma unroll 1
        for (int jb = 8; jb < K; jb += 8) {
            T g[4][CPT];
            products(jb, g, true);
            products(jb + 4, g, false);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    T y = g[i][cc] - comp[i][cc];
                    T t = out[i][cc] + y;
                    comp[i][cc] = (t - out[i][cc]) - y;
                    out[i][cc] = t;
                }
        }
    } else {
#pragma unroll 1
        for (int jb = 0; jb < K; jb += 4) products(jb, out, false);
    }
    if (COMP) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) out[i][cc] -= comp[i][cc];
    }
}

// E^T of a branch [K][K] into shared memory with rows of LDN, asynchronously (the caller commits
// and waits)
template <typename T, int THREADS>
__device__ inline void stage_rows(T *dst, const T *src, int tid)
{
    constexpr int V = 16 / sizeof(T);          // entries of one 16-byte copy
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int f = tid; f < K2 / V; f += THREADS) {
        const int r = f / (K / V), c = (f - r * (K / V)) * V;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + (uint32_t)((r * LDN + c) * sizeof(T))),
                     "l"(src + (size_t)r * K + c) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// What the children of a node need, into the two buffers at Et (K2 entries each), asynchronously
// (committed; the caller waits): an internal child's E^T as it is, and for a leaf child the row of
// its E^T that each tile column selects, one row of 64 states per column (the column's row read in
// one piece; a thread that gathers its four states from global memory touches a line per column:
// two thirds of the kernel's L1 wavefronts).  The 16-byte chunks of a row are permuted by XOR with
// the number of the thread column that reads it, so that those reads are free of conflicts.
template <typename T, int TC, int CPT, int THREADS>
__device__ inline void stage_children(T *Et, const T *Pbase, const SchedNode &nx, const uint8_t *lvT, int tid)
{
    constexpr int V = 16 / sizeof(T), NC = K / V;
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const int child = side ? nx.rc : nx.lc;
        const T *src = Pbase + (size_t)child * K2;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Et + side * K2);
        if ((side ? nx.rslot : nx.lslot) < 0) {
            for (int f = tid; f < TC * NC; f += THREADS) {
                const int col = f / NC, ch = f % NC;
                const int s = lvT[child * TC + col];
                if (s < K)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                 :: "r"(dst + (uint32_t)(col * NC + (ch ^ (4 / V * ((col / CPT) & 15)))) * 16),
                                    "l"(src + s * K + ch * V) : "memory");
            }
        } else {
            for (int f = tid; f < K * NC; f += THREADS)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16 * f), "l"(src + f * V) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Partial of child c at its parent: v[a] = alpha_c[a] + sum_j E_c[a][j] alpha_c[j]
// (internal child, slot >= 0; Et = E_c^T) or the gather v[a] = P_c[a][s] of a
// leaf in state s (1 for a marginalised leaf: P rows sum to 1).
template <typename T, int TC, int KAHAN, int CPT = TC / 16, int UNROLL = 1>
__device__ inline void child_partial(const T *Et, const T *slots, int slot, int leaf, const uint8_t *lvT, int a0,
                                     int c0, T v[4][CPT], int64_t dither_col0 = -1, bool staged = false,
                                     const float *dlo = nullptr)
{
    // dlo (may be null): the low parts of this branch's diag(E), added to the diagonal
    // term: FP32 storage of E_ii is the one rounding that every column sharing a state
    // at this node repeats identically, so over a long region it adds up coherently
    // (2-3e-3 dB over 10,000 codons at rho = 3 without it)
    if (slot < 0) {
        if (staged) {   // the columns' rows of the leaf's E^T, as stage_children placed them
            constexpr int V = 16 / sizeof(T);
            const int ch = (a0 / V) ^ (4 / V * ((c0 / CPT) & 15));
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) {
                const int s = lvT[leaf * TC + c0 + cc];
                const T c = (dither_col0 >= 0) ? (T)(1.0f + (float)dither_k(dither_col0 + c0 + cc, leaf) * (1.0f / 256.0f))
                                               : (T)1;
                T e[4];
                Vec4<T>::load(Et + (c0 + cc) * K + ch * V, e);
                // only the thread that holds state s needs the diagonal's low part
                const T lo_s = (dlo && s >= a0 && s < a0 + 4 && s < K) ? (T)dlo[s] : (T)0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int a = a0 + i;
                    T val = fma(e[i], c, (a == s ? c : (T)0));
                    if (a == s) {       // + c lo_s: the rounding error r of c (1 + E_ss) is recovered (exactly
                                        // when P_ss >= 1/2, where c - val is exact), so that lo_s enters
                                        // the one final rounding instead of vanishing below half an ulp of c
                        const T r = fma(e[i], c, c - val);
                        val = val + fma(lo_s, c, r);
                    }
                    v[i][cc] = (s >= K) ? c : val;
                }
            }
            return;
        }
#pragma unroll
        for (int cc = 0; cc < CPT; cc++) {
            int s = lvT[leaf * TC + c0 + cc];
            // with dithering, c * P[a][s] in one rounding (c exact, see dither_k)
            const T c = (dither_col0 >= 0) ? (T)(1.0f + (float)dither_k(dither_col0 + c0 + cc, leaf) * (1.0f / 256.0f))
                                           : (T)1;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int a = a0 + i;
                v[i][cc] = (s >= K) ? c : fma(Et[s * K + a], c, (a == s ? c : (T)0));
            }
        }
        return;
    }
    const T *al = slots + (size_t)slot * K * TC;
    contract<T, TC, KAHAN, CPT, UNROLL>(Et, al, a0, c0, v);
    T lo[4] = {(T)0, (T)0, (T)0, (T)0};
    if (dlo) {
        const float4 l4 = *reinterpret_cast<const float4 *>(dlo + a0);
        lo[0] = (T)l4.x; lo[1] = (T)l4.y; lo[2] = (T)l4.z; lo[3] = (T)l4.w;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        T x[CPT];
        ColLoad<T, CPT>::load(al + (a0 + i) * TC + c0, x);
#pragma unroll
        for (int cc = 0; cc < CPT; cc++) v[i][cc] = x[cc] + (dlo ? fma(lo[i], x[cc], v[i][cc]) : v[i][cc]);
    }
}

}  // namespace pcsf
