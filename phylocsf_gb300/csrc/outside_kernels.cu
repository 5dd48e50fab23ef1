// Outside-pass products beyond the gradient: the expected substitution counts of
// every branch (the sufficient statistics of PhyloEM) and the posterior state
// distribution of selected nodes at every column.
//
// Reference mathematics (paths relative to mlin/PhyloCSF):
//   outside pass             lib/CamlPaml/PhyloLik.ml:96-120    beta_i = P_i^T (beta_p . (P_s alpha_s))
//   node posterior           lib/CamlPaml/PhyloLik.ml:127-138   alpha_i . beta_i / z (a leaf: its own vector)
//   branch posteriors        lib/CamlPaml/PhyloLik.ml:140-174   beta_p[a] (P_s alpha_s)[a] P_i[a][b] alpha_i[b] / z
//   sufficient statistics    lib/CamlPaml/PhyloEM.ml:14-20      the branch posteriors summed over the columns
// With inter_c = beta_p . v_s (v_s = P_s alpha_s the sibling's partial at the parent),
// the counts of branch c are P_c[a][b] M_c[a][b] with M_c = sum_col inter_c alpha_c^T / z:
// per tile a 64 x 64 x (tile columns) product, accumulated over the tiles of a region
// and multiplied by P_c once at the end.
//
// One CTA owns one column tile at a time and leaves its count product in memory of the tile's own;
// k_counts adds the tiles of a request in order in FP64 and multiplies by P_c (no atomics): the results
// depend on the region alone, not on the launch configuration or on the call's other regions.  A CTA
// per request, its tiles in a row, left a call of 64 regions waiting for the longest one, 47 tiles
// (38.4 ms on 29 leaves, 27,641 columns, where the count products also read alpha from global memory
// with 16 lines per load; now the products' operands lie column by column in shared memory).
// Measured there: 1.4 ms, and 1.1 of k_counts.  What bounds it is the chain of a side's phases at three
// CTAs per SM, and in k_counts FP64 conversions and sums (two lanes per clock).
// The inside pass is the one of k_grad and
// stores every child partial, the alpha of every internal node and the per-column
// exponents of the power-of-two rescaling in a per-CTA scratch area; exponent
// bookkeeping per column as in k_grad:
//   alpha_i = alpha~_i 2^{e(i)},  beta_c = beta~_c 2^{f(c)},  z = z~ 2^{e(root)}.
// FP64 on the FP64 engine; FP32 with compensated sums on the others.
#include <algorithm>
#include <cmath>

#include "pcsf_internal.h"
#include "prune_common.cuh"

namespace pcsf {

namespace {

constexpr int OS_THREADS = 256;
constexpr int OS_TC = 32;
constexpr int OS_CPT = OS_TC / 16;

template <typename T>
struct OutLayout {
    static size_t smem(int nslots, int nl, int nint)
    {
        // Mat[2], slots, X; in the outside pass E^T (rows of LDN) and the two transposed tiles take their place
        size_t b = sizeof(T) * (std::max<size_t>(2 * (size_t)K2 + (size_t)nslots * K * OS_TC, (size_t)K * LDN + 2 * OS_TC * LDN) +
                                (size_t)K * OS_TC);
        b += sizeof(typename AtomMax<T>::U) * OS_TC;                                               // column maxima
        b += sizeof(double) * 2 * OS_TC;                                                           // z~, column weights
        b += sizeof(int) * OS_TC;                                                                  // e(root)
        b += sizeof(SchedNode) * nint;
        b = (b + 15) & ~size_t(15);
        b += (size_t)nl * OS_TC;
        return (b + 15) & ~size_t(15);
    }
    static size_t scratch(int nl)
    {
        const int n = 2 * nl - 1;
        size_t b = sizeof(T) * ((size_t)(n - 1) + 2 * (size_t)(nl - 1)) * K * OS_TC;   // V, alpha~ and beta~ of internal nodes
        b += sizeof(int) * 2 * (size_t)n * OS_TC;                                      // e, f
        return (b + 255) & ~size_t(255);
    }
};

template <typename T, int KAHAN>
__global__ void __launch_bounds__(OS_THREADS) k_outside(OutsideArgs a)
{
    constexpr int TC = OS_TC, CPT = OS_CPT;
    typedef typename AtomMax<T>::U MU;
    extern __shared__ __align__(16) unsigned char osm[];
    T *Mat = reinterpret_cast<T *>(osm);                           // [2][K][K]
    T *slots = Mat + 2 * K2;                                        // [nslots][K][TC]
    // outside pass: E^T of a branch, and inter and alpha column by column (the inside pass's
    // Mat and slots are idle then)
    T *Ert = Mat, *XT = Mat + K * LDN, *YT = XT + TC * LDN;         // [K][LDN], [TC][LDN], [TC][LDN]
    constexpr size_t OUT = (size_t)K * LDN + 2 * TC * LDN;
    const size_t inw = 2 * (size_t)K2 + (size_t)a.nslots * K * TC;
    T *X = Mat + (inw > OUT ? inw : OUT);                           // [K][TC]
    MU *colmax = reinterpret_cast<MU *>(X + K * TC);                // [TC]
    double *zt = reinterpret_cast<double *>(colmax + TC);           // [TC]
    double *wcol = zt + TC;                                         // [TC]
    int *eroot = reinterpret_cast<int *>(wcol + TC);                // [TC]
    SchedNode *sched = reinterpret_cast<SchedNode *>(eroot + TC);   // [n_internal]
    size_t off = (reinterpret_cast<unsigned char *>(sched + a.n_internal) - osm + 15) & ~size_t(15);
    uint8_t *lvT = osm + off;                                       // [nl][TC]
    __shared__ double wsum[OS_THREADS / 32];

    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;
    const int a0 = 4 * ty, c0 = CPT * tx;     // contraction tiles: 4 states x 2 columns
    const int b0 = 4 * tx;                     // count blocks: states a0.. (from) x b0.. (to)
    const int nl = a.nl, n = 2 * nl - 1, root = n - 1;
    unsigned char *sbase = reinterpret_cast<unsigned char *>(a.scratch) + (size_t)blockIdx.x * a.scratch_per_cta;
    T *V = reinterpret_cast<T *>(sbase);                             // [n-1][K][TC]
    T *A = V + (size_t)(n - 1) * K * TC;                             // [nl-1][K][TC] alpha~ (internal nodes)
    T *B = A + (size_t)(nl - 1) * K * TC;                            // [nl-1][K][TC] beta~ (internal nodes)
    int *eS = reinterpret_cast<int *>(B + (size_t)(nl - 1) * K * TC);   // [n][TC]
    int *fS = eS + (size_t)n * TC;                                   // [n][TC]
    auto e_of = [&](int node, int col) -> int { return node < nl ? 0 : eS[(size_t)node * TC + col]; };

    for (int f = tid; f < a.n_internal; f += OS_THREADS) sched[f] = a.sched[f];

    for (int w = a.wi0 + blockIdx.x; w < a.wi1; w += gridDim.x) {
        const WorkItem wi = a.wi[w];
        const Request rq = a.req[wi.request];
        const int md = rq.model;
        const T *Pbase = reinterpret_cast<const T *>(a.Pbuf) + (size_t)rq.pset * a.nbr * K2;
        const double *pr = a.m.prior + md * K;
        T *cnt = a.counts ? reinterpret_cast<T *>(a.tile_counts) + (size_t)(w - a.wi0) * a.nbr * K2 : nullptr;
        const int ncols = wi.ncols;
        const uint8_t *lg = a.leaves + (size_t)wi.col0 * nl;
        __syncthreads();   // the previous tile is finished with shared memory
        for (int f = tid; f < TC * nl; f += OS_THREADS) {
            const int c = f / nl, l = f - c * nl;
            lvT[l * TC + c] = (c < ncols) ? lg[f] : (uint8_t)K;
        }
        for (int f = tid; f < TC; f += OS_THREADS) colmax[f] = 0;

        // ---------------- inside pass, storing the child partials and the node alphas
        __syncthreads();   // leaf states ready
        stage_children<T, TC, CPT, OS_THREADS>(Mat, Pbase, sched[0], lvT, tid);
        for (int ni = 0; ni < a.n_internal; ni++) {
            const SchedNode sn = sched[ni];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            T vl[4][CPT], vr[4][CPT];
            child_partial<T, TC, KAHAN>(Mat, slots, sn.lslot, sn.lc, lvT, a0, c0, vl, -1, true);
            child_partial<T, TC, KAHAN>(Mat + K2, slots, sn.rslot, sn.rc, lvT, a0, c0, vr, -1, true);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    V[((size_t)sn.lc * K + a0 + i) * TC + c0 + cc] = vl[i][cc];
                    V[((size_t)sn.rc * K + a0 + i) * TC + c0 + cc] = vr[i][cc];
                }
            __syncthreads();   // Mat and slot reads done
            if (ni + 1 < a.n_internal) stage_children<T, TC, CPT, OS_THREADS>(Mat, Pbase, sched[ni + 1], lvT, tid);
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) {
                T mx = (T)0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    vl[i][cc] *= vr[i][cc];
                    mx = vl[i][cc] > mx ? vl[i][cc] : mx;
                }
                AtomMax<T>::upd(colmax + c0 + cc, mx);
            }
            __syncthreads();
            T *out = slots + (size_t)sn.oslot * K * TC;
            T *Ai = A + (size_t)(sn.node - nl) * K * TC;
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) {
                const T mx = AtomMax<T>::get(colmax + c0 + cc);
                const int e = (mx > (T)0) ? exp_of(mx) : 0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const T y = scale2(vl[i][cc], -e);
                    out[(a0 + i) * TC + c0 + cc] = y;
                    Ai[(size_t)(a0 + i) * TC + c0 + cc] = y;
                }
                if (ty == 0) {
                    const int col = c0 + cc;
                    eS[(size_t)sn.node * TC + col] = e_of(sn.lc, col) + e_of(sn.rc, col) + e;
                }
            }
            __syncthreads();   // colmax reads done
            for (int f = tid; f < TC; f += OS_THREADS) colmax[f] = 0;
        }
        __syncthreads();
        // ---------------- root: z~ and the column log-likelihoods
        double tl = 0.0;
        if (tid < TC) {
            const T *ar = A + (size_t)(root - nl) * K * TC;
            double z = 0.0;
            for (int s = 0; s < K; s++) z += (double)ar[s * TC + tid] * pr[s];
            zt[tid] = z;
            eroot[tid] = eS[(size_t)root * TC + tid];
            if (tid < ncols) tl = (z > 0.0) ? log(z) + (double)eroot[tid] * 0.69314718055994530942 : -INFINITY;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tl += __shfl_down_sync(0xffffffffu, tl, o);
        if ((tid & 31) == 0) wsum[tid >> 5] = tl;
        {   // beta~_root = prior, f(root) = 0
            T *Br = B + (size_t)(root - nl) * K * TC;
            for (int f = tid; f < K * TC; f += OS_THREADS) Br[f] = (T)pr[f / TC];
            for (int f = tid; f < TC; f += OS_THREADS) fS[(size_t)root * TC + f] = 0;
        }
        __syncthreads();
        if (tid == 0) {
            double lpr = 0.0;
            for (int k = 0; k < (TC + 31) / 32; k++) lpr += wsum[k];
            a.tile_lpr[w] = lpr;
        }
        // posteriors of the selected root and leaves (node_posterior: zeros where z = 0)
        if (a.sel) {
            const int kr = a.sel[root];
            if (kr >= 0) {
                const T *ar = A + (size_t)(root - nl) * K * TC;
                for (int f = tid; f < K * TC; f += OS_THREADS) {
                    const int x = f / TC, col = f % TC;
                    if (col >= ncols) continue;
                    const double z = zt[col];
                    a.post[((size_t)kr * a.total_cols + wi.col0 + col) * K + x] =
                        (z > 0.0) ? (double)ar[x * TC + col] * pr[x] / z : 0.0;
                }
            }
            for (int l = 0; l < nl; l++) {
                const int kl = a.sel[l];
                if (kl < 0) continue;
                for (int f = tid; f < K * TC; f += OS_THREADS) {
                    const int x = f / TC, col = f % TC;
                    if (col >= ncols) continue;
                    const int s = lvT[l * TC + col];
                    a.post[((size_t)kl * a.total_cols + wi.col0 + col) * K + x] =
                        (zt[col] > 0.0) ? ((s >= K || s == x) ? 1.0 : 0.0) : 0.0;
                }
            }
        }

        // ---------------- outside pass, parents before children
        for (int ni = a.n_internal - 1; ni >= 0; ni--) {
            const SchedNode sn = sched[ni];
            const int p = sn.node;
            const T *Bp = B + (size_t)(p - nl) * K * TC;
            for (int side = 0; side < 2; side++) {
                const int c = side ? sn.rc : sn.lc;
                const int s = side ? sn.lc : sn.rc;
                const bool internal = c >= nl;
                __syncthreads();   // the previous side is finished with X, Mat[0], colmax, wcol
                if (internal) stage_rows<T, OS_THREADS>(Ert, Pbase + (size_t)c * K2, tid);
                for (int f = tid; f < TC; f += OS_THREADS) colmax[f] = 0;
                const T *Vs = V + (size_t)s * K * TC;
                for (int f = tid; f < K * TC; f += OS_THREADS) X[f] = Bp[f] * Vs[f];    // inter~
                if (tid < TC) {   // weight of column tid in the counts: 2^{f(p) + e(s) + e(c) - e(root)} / z~
                    const double z = zt[tid];
                    wcol[tid] = (tid < ncols && z > 0.0)
                                    ? ldexp(1.0, fS[(size_t)p * TC + tid] + e_of(s, tid) + e_of(c, tid) - eroot[tid]) / z
                                    : 0.0;
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                if (internal) {
                    // beta~_c = P_c^T inter~ = inter~ + E_c^T inter~, rescaled per column
                    T bt[4][CPT];
                    contract_rows<T, TC, KAHAN>(Ert, X, a0, c0, bt);
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        T mx = (T)0;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            bt[i][cc] += X[(a0 + i) * TC + c0 + cc];
                            mx = bt[i][cc] > mx ? bt[i][cc] : mx;
                        }
                        AtomMax<T>::upd(colmax + c0 + cc, mx);
                    }
                    __syncthreads();
                    T *Bc = B + (size_t)(c - nl) * K * TC;
                    const T *Ac = A + (size_t)(c - nl) * K * TC;
                    const int kc = a.sel ? a.sel[c] : -1;
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        const int col = c0 + cc;
                        const T mx = AtomMax<T>::get(colmax + col);
                        const int e = (mx > (T)0) ? exp_of(mx) : 0;
                        const int fc = fS[(size_t)p * TC + col] + e_of(s, col) + e;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const T y = scale2(bt[i][cc], -e);
                            Bc[(size_t)(a0 + i) * TC + col] = y;
                            if (kc >= 0 && col < ncols) {
                                const double z = zt[col];
                                a.post[((size_t)kc * a.total_cols + wi.col0 + col) * K + a0 + i] =
                                    (z > 0.0) ? ldexp((double)Ac[(size_t)(a0 + i) * TC + col] * (double)y,
                                                      e_of(c, col) + fc - eroot[col]) / z
                                              : 0.0;
                            }
                        }
                        if (ty == 0) fS[(size_t)c * TC + col] = fc;
                    }
                }
                if (cnt) {
                    // inter~ w and alpha~_c, column by column (from here a column's 64 states
                    // are contiguous: one vector load for each of a thread's two sides)
                    const T *Ac = A + (size_t)(internal ? c - nl : 0) * K * TC;
                    for (int f = tid; f < K * TC; f += OS_THREADS) {
                        XT[(f % TC) * LDN + f / TC] = (T)((double)X[f] * wcol[f % TC]);
                        if (internal) YT[(f % TC) * LDN + f / TC] = Ac[f];
                    }
                    __syncthreads();
                    // M_c[a][b] += sum_col inter~[a] w alpha~_c[b] for this thread's 4 x 4 block
                    T acc[4][4];
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[i][j] = (T)0;
                    if (internal) {
#pragma unroll 4
                        for (int col = 0; col < TC; col++) {
                            T xa[4], yb[4];
                            Vec4<T>::load(XT + col * LDN + a0, xa);
                            Vec4<T>::load(YT + col * LDN + b0, yb);
#pragma unroll
                            for (int i = 0; i < 4; i++)
#pragma unroll
                                for (int j = 0; j < 4; j++) acc[i][j] += xa[i] * yb[j];
                        }
                    } else {
#pragma unroll 4
                        for (int col = 0; col < TC; col++) {
                            const int sl = lvT[c * TC + col];
                            T xa[4];
                            Vec4<T>::load(XT + col * LDN + a0, xa);
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                const bool hit = sl >= K || sl == b0 + j;
#pragma unroll
                                for (int i = 0; i < 4; i++) acc[i][j] = hit ? acc[i][j] + xa[i] : acc[i][j];
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) ColStore<T, 4>::store(cnt + (size_t)c * K2 + (a0 + i) * K + b0, acc[i]);
                }
            }
        }
    }
}

// Request r's tiles of this launch, in order, onto the sums of those before: the log-likelihood and
// sum M_c, which the request's last tile makes counts = P_c o sum M_c.  One CTA per (branch, request).
template <typename T>
__global__ void __launch_bounds__(OS_THREADS) k_counts(OutsideArgs a)
{
    const int c = blockIdx.y, r = blockIdx.x, tid = threadIdx.x;
    const int b0 = a.wi_begin[r], b1 = a.wi_begin[r + 1], w0 = max(b0, a.wi0), w1 = min(b1, a.wi1);
    // nothing of this request in this launch (an empty one has its zeros from the first)
    if (w0 >= w1 && (b0 < b1 || a.wi0 > 0)) return;
    const bool first = b0 >= a.wi0, last = b1 <= a.wi1;
    if (c == 0 && tid == 0) {
        double lpr = first ? 0.0 : a.lpr[r];
        for (int w = w0; w < w1; w++) lpr += a.tile_lpr[w];
        a.lpr[r] = lpr;
    }
    if (!a.counts) return;
    const T *Et = reinterpret_cast<const T *>(a.Pbuf) + ((size_t)a.req[r].pset * a.nbr + c) * K2;
    const T *tc = reinterpret_cast<const T *>(a.tile_counts) + (size_t)c * K2;
    double *out = a.counts + ((size_t)r * a.nbr + c) * K2;
    for (int f = tid; f < K2; f += OS_THREADS) {
        const int aa = f / K, bb = f % K;
        double m = first ? 0.0 : out[f];
        for (int w = w0; w < w1; w++) m += (double)tc[(size_t)(w - a.wi0) * a.nbr * K2 + f];
        out[f] = last ? m * ((double)Et[bb * K + aa] + (aa == bb ? 1.0 : 0.0)) : m;
    }
}

template <typename T, int KAHAN>
cudaError_t launch_outside_t(const OutsideArgs &a, cudaStream_t s, int grid)
{
    const size_t smem = OutLayout<T>::smem(a.nslots, a.nl, a.n_internal);
    cudaError_t e = allow_smem<k_outside<T, KAHAN>>();
    if (e != cudaSuccess) return e;
    if (a.wi1 > a.wi0) k_outside<T, KAHAN><<<std::min(grid, a.wi1 - a.wi0), OS_THREADS, smem, s>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_counts<T><<<dim3(a.nreq, a.counts ? a.nbr : 1), OS_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int KAHAN>
int ctas_per_sm_t(int nslots, int nl, int nint)
{
    const size_t smem = OutLayout<T>::smem(nslots, nl, nint);
    int n = 0;
    if (allow_smem<k_outside<T, KAHAN>>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_outside<T, KAHAN>, OS_THREADS, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return std::max(n, 1);
}

}  // namespace

int outside_tile_cols() { return OS_TC; }

int outside_ctas_per_sm(bool fp64, int comp, int nslots, int nl, int nint)
{
    if (fp64) return ctas_per_sm_t<double, 0>(nslots, nl, nint);
    return comp == 2 ? ctas_per_sm_t<float, 2>(nslots, nl, nint) : ctas_per_sm_t<float, 1>(nslots, nl, nint);
}

size_t outside_smem_bytes(bool fp64, int nslots, int nl, int nint)
{
    return fp64 ? OutLayout<double>::smem(nslots, nl, nint) : OutLayout<float>::smem(nslots, nl, nint);
}

size_t outside_scratch_per_cta(bool fp64, int nl)
{
    return fp64 ? OutLayout<double>::scratch(nl) : OutLayout<float>::scratch(nl);
}

cudaError_t launch_outside(bool fp64, int comp, const OutsideArgs &a, cudaStream_t s, int grid)
{
    if (a.nreq <= 0) return cudaSuccess;
    if (fp64) return launch_outside_t<double, 0>(a, s, grid);
    if (comp == 2) return launch_outside_t<float, 2>(a, s, grid);
    return launch_outside_t<float, 1>(a, s, grid);
}

}  // namespace pcsf
