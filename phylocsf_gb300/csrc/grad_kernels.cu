// Adjoint (outside-pass) gradient of the log-likelihood with respect to every
// branch length, for a batch of (region, model, rho) requests.
//
// Reference mathematics (paths relative to mlin/PhyloCSF):
//   outside pass          lib/CamlPaml/PhyloLik.ml:96-120   beta_i = P_i^T (beta_p . (P_s alpha_s))
//   branch posteriors     lib/CamlPaml/PhyloLik.ml:140-174
//   dP/dt                 lib/CamlPaml/Q.ml:260-275          dP/dt = Q P(t)
//   d ELL / d branch      lib/CamlPaml/PhyloEM.ml:140-171    (Fisher identity: = d logL / d t)
// Per column, with v_c = P_c alpha_c the partial of child c at its parent p and
// s its sibling:
//   inter_c = beta_p . v_s,   d log z / d t_c = inter_c^T Q v_c / z,   beta_c = P_c^T inter_c.
//
// One CTA (256 threads) owns a tile of 32 columns, two CTAs share an SM.  The inside pass is
// the one of k_prune (a node's operands copied one node ahead) but also stores the partial v_c of every child and the per-column exponents of the
// power-of-two rescaling in a per-CTA global scratch area; the outside pass then walks the
// schedule in reverse.  A leaf child's partial is one gathered row of E^T plus the identity
// (P_c[a][s]); with RECOMP the outside pass recomputes it from the leaf state instead of
// storing it (a third less scratch, the same values, a few percent more time for the
// scattered re-reads of E^T rows).  Exponent bookkeeping per column:
// alpha_i = alpha~_i 2^{e(i)} with e(i) = e(l) + e(r) + s_i, beta_c = beta~_c 2^{f(c)}
// with f(c) = f(p) + e(s) + t_c, and the gradient term carries
// 2^{f(p) + e(s) + e(c) - e(root)} against the scaled z~.
//
// What bounds it: the FP32 contractions (two per internal branch, one per leaf branch, and
// three or four more with the rate parameters), about half of the time.  The rest was the
// chain around them: 64-column tiles left one CTA per SM, E^T was transposed into shared
// memory with 32-way bank conflicts, and each side ended in 16 FP64 additions, an ldexp and
// a division on two of the eight warps (an SM issues two FP64 lanes per clock).  Now E^T is
// contracted as stored, a column's weight 2^ex / z~ is formed once ahead by one warp, all
// eight warps share the FP64 sums of a side, and these run beside the next side's
// contractions; the warps' sums meet in shared memory one side later, so that a tile leaves one
// row of sums (a row per warp took eight times the memory, and k_reduce_grad eight times as many
// dependent additions).  Measured, per column: 58 leaves 173 -> 88 ns, 100 leaves with two rate
// parameters 955 -> 387 ns.
#include <algorithm>
#include <cmath>

#include "pcsf_internal.h"
#include "prune_common.cuh"

namespace pcsf {

constexpr int GR_THREADS = 256;
constexpr int GR_WARPS = GR_THREADS / 32;
constexpr int GR_UNROLL = 3;         // blocks of a contraction in a row (see contract_pairs)
constexpr int GR_TC = 32;            // columns per tile

template <typename T, bool RECOMP>
struct GradLayout {
    static constexpr int TC = GR_TC;
    // shared memory: Q, [U], then a region that holds the inside pass's slots and E^T (with the
    // rate parameters E^T sits where Q and U go afterwards: two CTAs per SM on 100 leaves), and in
    // the outside pass E^T (rows of LDN), [H_x^T and two tiles,] and X
    __host__ __device__ static size_t region(int nslots, int npar)
    {
        const size_t in = (npar ? 0 : 2 * (size_t)K2) + (size_t)nslots * K * TC;
        const size_t out = (size_t)K * LDN + (size_t)K * TC + (npar ? (size_t)K2 + 2 * (size_t)K * TC : 0);
        return in > out ? in : out;
    }
    // [2][1 + npar][16][TC] column sums; the root's [2][warps][TC] FP64 sums share the space
    __host__ __device__ static size_t reds(int npar)
    {
        const size_t r = 2 * (size_t)(1 + npar) * 16 * TC, z = 2 * GR_WARPS * TC * sizeof(double) / sizeof(T);
        return r > z ? r : z;
    }
    static size_t smem(int nslots, int nl, int nint, int npar)
    {
        size_t b = sizeof(T) * ((size_t)K2 + (npar ? (size_t)K2 + 3 * K : 0) + region(nslots, npar) + reds(npar));
        b += sizeof(double) * (3 * TC + 2 * (1 + npar) * GR_WARPS);
        b += sizeof(typename AtomMax<T>::U) * 2 * TC + sizeof(int) * ((npar ? 4 : 5) * TC + (size_t)nslots * TC);
        b += sizeof(SchedNode) * nint;
        b = (b + 15) & ~size_t(15);
        b += (size_t)nl * TC;
        return (b + 15) & ~size_t(15);
    }
    // stored child partials: every child's (n - 1), or with RECOMP the internal children's
    __host__ __device__ static size_t nv(int nl) { return RECOMP ? (size_t)(nl - 1) : (size_t)(2 * nl - 2); }
    __host__ __device__ static size_t scratch(int nl, int npar)
    {
        const int n = 2 * nl - 1;
        size_t b = sizeof(T) * (nv(nl) + (nl - 1)) * K * TC;        // child partials, betas
        b += sizeof(int) * 2 * (size_t)n * TC;
        b = (b + 255) & ~size_t(255);
        if (npar) b += (sizeof(T) * (size_t)(nl - 1) * K * TC + 255) & ~size_t(255);   // alpha of internal nodes
        return b;
    }
};

template <typename T, int KAHAN, bool RECOMP>
__global__ void __launch_bounds__(GR_THREADS, sizeof(T) == 4 ? 2 : 1) k_grad(GradArgs a)
{
    typedef GradLayout<T, RECOMP> Layout;
    constexpr int TC = GR_TC, CPT = TC / 16;
    typedef typename AtomMax<T>::U MU;
    extern __shared__ __align__(16) unsigned char gsm[];
    const int npar = a.npar;
    T *Qs = reinterpret_cast<T *>(gsm);                            // [K][K] Q row-major
    T *Us = Qs + K2;                                                // [K][K] U row-major (npar)
    T *isT = Us + (npar ? K2 : 0), *sqT = isT + (npar ? K : 0), *wmT = sqT + (npar ? K : 0);   // [K] each (npar)
    T *R = wmT + (npar ? K : 0);
    T *Mat = npar ? Qs : R, *slots = npar ? R : R + 2 * K2;         // inside: [2][K][K], [nslots][K][TC]
    T *Er = R, *X = R + K * LDN;                                    // outside: [K][LDN], [K][TC]
    T *Hb = X + K * TC, *Q1 = Hb + K2, *Q2 = Q1 + K * TC;           // [K][K], [K][TC] x 2 (npar)
    T *red = R + Layout::region(a.nslots, npar);                    // [2][1 + npar][16][TC]
    double *zp = reinterpret_cast<double *>(red);                   // root: [2][GR_WARPS][TC]
    double *zt = reinterpret_cast<double *>(red + Layout::reds(npar));   // [TC] 1 / z~ (0: no gradient)
    double *wcol = zt + TC;                                         // [2][TC] column weights 2^ex / z~
    double *wsum = wcol + 2 * TC;                                   // [2][1 + npar][GR_WARPS] a side's sums of each warp
    MU *colmax = reinterpret_cast<MU *>(wsum + 2 * (1 + npar) * GR_WARPS);    // [2][TC]
    int *eroot = reinterpret_cast<int *>(colmax + 2 * TC);          // [TC]
    int *ebase = eroot + TC;                                        // [2][TC] f(p) + e(s), by side: one side's is read
                                                                    //   (by half a warp) while the next side's is written
                                                                    //   (npar: a barrier apart, [TC] for both)
    int *wexp = ebase + (npar ? 1 : 2) * TC;                        // [2][TC] the weight's exponent where 2^ex / z~ may not be normal, else 0
    int *slexp = wexp + 2 * TC;                                        // [nslots][TC] exponents of the slots' partials
    SchedNode *sched = reinterpret_cast<SchedNode *>(slexp + a.nslots * TC);   // [n_internal]
    size_t off = (reinterpret_cast<unsigned char *>(sched + a.n_internal) - gsm + 15) & ~size_t(15);
    uint8_t *lvT = gsm + off;                                       // [nl][TC]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ty = tid / 16, tx = tid % 16;
    const int a0 = 4 * ty, c0 = CPT * tx;
    const int nl = a.nl, n = 2 * nl - 1;
    unsigned char *sbase = reinterpret_cast<unsigned char *>(a.scratch) + (size_t)blockIdx.x * a.scratch_per_cta;
    T *V = reinterpret_cast<T *>(sbase);                             // [nv][K][TC] child partials (vslot)
    T *B = V + Layout::nv(nl) * K * TC;                              // [nl-1][K][TC] (internal nodes)
    int *eS = reinterpret_cast<int *>(B + (size_t)(nl - 1) * K * TC);  // [n][TC]
    int *fS = eS + (size_t)n * TC;                                   // [n][TC]
    T *Ascr = reinterpret_cast<T *>(sbase + ((sizeof(T) * (Layout::nv(nl) + (nl - 1)) * K * TC +
                                              sizeof(int) * 2 * (size_t)n * TC + 255) & ~size_t(255)));   // [nl-1][K][TC]
    // a child's slab among the stored partials (RECOMP: internal children only)
    auto vslot = [&](int c) -> size_t { return RECOMP ? (size_t)(c - nl) : (size_t)c; };
    const int gstride = a.nbr + npar;
    auto e_of = [&](int node, int col) -> int { return node < nl ? 0 : eS[(size_t)node * TC + col]; };
    // partial of a RECOMP leaf child c, state st, tile column col: exactly as the inside pass
    // formed it (E^T[s][st] + delta, in one rounding; 1 for a marginalised leaf)
    auto leaf_part = [&](const T *Pbase, int c, int st, int col) -> T {
        const int sl = lvT[c * TC + col];
        if (sl >= K) return (T)1;
        return fma(Pbase[(size_t)c * K2 + (size_t)sl * K + st], (T)1, sl == st ? (T)1 : (T)0);
    };

    for (int f = tid; f < a.n_internal; f += GR_THREADS) sched[f] = a.sched[f];

    for (int w = blockIdx.x; w < a.nwi; w += gridDim.x) {
        const WorkItem wi = a.wi[w];
        const Request rq = a.req[wi.request];
        const int md = rq.model;
        const T *Pbase = reinterpret_cast<const T *>(a.Pbuf) + (size_t)rq.pset * a.nbr * K2;
        const int ncols = wi.ncols;
        const uint8_t *lg = a.leaves + (size_t)wi.col0 * nl;
        double *gout = a.gpart + (size_t)w * gstride;
        __syncthreads();   // previous work item finished with shared memory
        for (int f = tid; f < TC * nl; f += GR_THREADS) {
            int c = f / nl, l = f - c * nl;
            lvT[l * TC + c] = (c < ncols) ? lg[f] : (uint8_t)K;
        }
        for (int f = tid; f < 2 * TC; f += GR_THREADS) colmax[f] = 0;

        // ---------------- inside pass, storing the child partials
        __syncthreads();       // leaf states ready
        stage_children<T, TC, CPT, GR_THREADS>(Mat, Pbase, sched[0], lvT, tid);
        for (int ni = 0; ni < a.n_internal; ni++) {
            const SchedNode sn = sched[ni];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            T vl[4][CPT], vr[4][CPT];
            child_partial<T, TC, KAHAN, CPT, GR_UNROLL>(Mat, slots, sn.lslot, sn.lc, lvT, a0, c0, vl, -1, true);
            child_partial<T, TC, KAHAN, CPT, GR_UNROLL>(Mat + K2, slots, sn.rslot, sn.rc, lvT, a0, c0, vr, -1, true);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (!RECOMP || sn.lc >= nl) ColStore<T, CPT>::store(V + (vslot(sn.lc) * K + a0 + i) * TC + c0, vl[i]);
                if (!RECOMP || sn.rc >= nl) ColStore<T, CPT>::store(V + (vslot(sn.rc) * K + a0 + i) * TC + c0, vr[i]);
            }
            __syncthreads();   // Mat and slot reads done
            if (ni + 1 < a.n_internal) stage_children<T, TC, CPT, GR_THREADS>(Mat, Pbase, sched[ni + 1], lvT, tid);
            MU *cm = colmax + (ni & 1) * TC, *cm_next = colmax + ((ni + 1) & 1) * TC;
            if (tid < TC) cm_next[tid] = 0;
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) {
                T mx = (T)0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    vl[i][cc] *= vr[i][cc];
                    mx = vl[i][cc] > mx ? vl[i][cc] : mx;
                }
                AtomMax<T>::upd(cm + c0 + cc, mx);
            }
            __syncthreads();
            T *out = slots + (size_t)sn.oslot * K * TC;
            int ecol[CPT];
#pragma unroll
            for (int cc = 0; cc < CPT; cc++) {
                const T mx = AtomMax<T>::get(cm + c0 + cc);
                ecol[cc] = (mx > (T)0) ? exp_of(mx) : 0;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                T y[CPT];
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) y[cc] = scale2(vl[i][cc], -ecol[cc]);
                ColStore<T, CPT>::store(out + (a0 + i) * TC + c0, y);
                if (npar) ColStore<T, CPT>::store(Ascr + ((size_t)(sn.node - nl) * K + a0 + i) * TC + c0, y);
            }
            if (ty == 0)
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    const int col = c0 + cc;
                    const int e = (sn.lslot < 0 ? 0 : slexp[sn.lslot * TC + col]) +
                                  (sn.rslot < 0 ? 0 : slexp[sn.rslot * TC + col]) + ecol[cc];
                    slexp[sn.oslot * TC + col] = e;
                    eS[(size_t)sn.node * TC + col] = e;
                }
        }
        __syncthreads();
        // ---------------- root: z~, lpr and elpr terms (eight states per thread, then per column)
        const int root = n - 1;
        {
            const T *ar = slots + (size_t)sched[a.n_internal - 1].oslot * K * TC;
            const double *pr = a.m.prior + md * K, *wl = a.m.wlog + md * K;
            double z = 0.0, wz = 0.0;
            for (int s = 8 * warp; s < 8 * warp + 8; s++) {
                const double x = (double)ar[s * TC + lane];
                z += x * pr[s];
                wz += x * wl[s];
            }
            zp[warp * TC + lane] = z;
            zp[(GR_WARPS + warp) * TC + lane] = wz;
            // beta~_root = prior, f(root) = 0
            T *Br = B + (size_t)(root - nl) * K * TC;
            for (int f = tid; f < K * TC; f += GR_THREADS) Br[f] = (T)pr[f / TC];
            for (int f = tid; f < TC; f += GR_THREADS) fS[(size_t)root * TC + f] = 0;
        }
        __syncthreads();
        if (warp == 0) {
            double z = 0.0, wz = 0.0;
            for (int q = 0; q < GR_WARPS; q++) {
                z += zp[q * TC + lane];
                wz += zp[(GR_WARPS + q) * TC + lane];
            }
            const int er = slexp[sched[a.n_internal - 1].oslot * TC + lane];
            zt[lane] = (lane < ncols && z > 0.0) ? 1.0 / z : 0.0;
            eroot[lane] = er;
            double tl = 0.0, te = 0.0;
            if (lane < ncols) {
                if (z > 0.0) {
                    tl = log(z) + (double)er * 0.69314718055994530942;
                    te = wz / z;
                } else {
                    tl = -INFINITY;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tl += __shfl_down_sync(0xffffffffu, tl, o);
                te += __shfl_down_sync(0xffffffffu, te, o);
            }
            if (lane == 0) {
                a.partials[2 * (size_t)w] = tl;
                a.partials[2 * (size_t)w + 1] = te;
            }
        }
        for (int f = tid; f < 2 * TC; f += GR_THREADS) colmax[f] = 0;
        {
            const T *Qg = reinterpret_cast<const T *>(a.Qrow) + (size_t)md * K2;
            for (int f = tid; f < K2; f += GR_THREADS) Qs[f] = Qg[f];
            if (npar) {
                const T *Ug = reinterpret_cast<const T *>(a.Umat) + (size_t)md * K2;
                for (int f = tid; f < K2; f += GR_THREADS) Us[f] = Ug[f];
                if (tid < K) {
                    isT[tid] = (T)a.m.isq[md * K + tid];
                    sqT[tid] = (T)a.m.sq[md * K + tid];
                }
                __syncthreads();
                // U^T D^1/2 1, the eigenbasis image of a marginalised leaf (the same in every column)
                for (int f = tid; f < K * TC; f += GR_THREADS) X[f] = sqT[f / TC];
                __syncthreads();
                T qv[4][CPT];
                contract<T, TC, KAHAN, CPT, GR_UNROLL>(Us, X, a0, c0, qv);
                if (tx == 0)
#pragma unroll
                    for (int i = 0; i < 4; i++) wmT[a0 + i] = qv[i][0];
            }
        }

        // ---------------- outside pass, parents before children
        // a side's column sums (FP32, 16 per column) are weighted and added over a warp's columns in
        // FP64 one side later, and over the warps two sides later: pc, qc = the branches that wait in
        // buffers pb, qb.  Warp x adds value x (0 the branch's, 1 and 2 the parameters').
        int pc = -1, pb = 0, qc = -1, qb = 0;
        double pacc = 0.0;                // parameter warp - 1's derivative (lane 0 of warps 1 and 2)
        auto flush = [&]() {
            if (qc >= 0 && warp <= npar) {
                double g = lane < GR_WARPS ? wsum[(qb * (1 + npar) + warp) * GR_WARPS + lane] : 0.0;
#pragma unroll
                for (int o = GR_WARPS / 2; o > 0; o >>= 1) g += __shfl_down_sync(0xffffffffu, g, o);
                if (lane == 0) {
                    if (warp == 0) gout[qc] = g;
                    else pacc += g;
                }
            }
            qc = pc;
            qb = pb;
            if (pc < 0) return;
            const double wv = wcol[pb * TC + lane];
            const int we = wexp[pb * TC + lane];
            for (int x = 0; x <= npar; x++) {
                const T *rd = red + (size_t)(pb * (1 + npar) + x) * 16 * TC + lane;
                double g = (double)rd[2 * warp * TC] + (double)rd[(2 * warp + 1) * TC];
                g = (we ? ldexp(g, we) : g) * wv;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) g += __shfl_down_sync(0xffffffffu, g, o);
                if (lane == 0) wsum[(pb * (1 + npar) + x) * GR_WARPS + warp] = g;
            }
            pc = -1;
        };
        int sidx = 0;
        for (int ni = a.n_internal - 1; ni >= 0; ni--) {
            const SchedNode sn = sched[ni];
            const int p = sn.node;
            const T *Bp = B + (size_t)(p - nl) * K * TC;
            __syncthreads();   // the betas of the last node are written, X and E^T are free
            if (ni > 0) {      // the next node's slabs, from DRAM into L2 (69,983 columns, 58 leaves: 6.61 -> 6.40 ms)
                const SchedNode nx = sched[ni - 1];
                constexpr int NL = K * TC * sizeof(T) / 128;
                for (int f = tid; f < 3 * NL; f += GR_THREADS) {
                    const int c = f < NL ? nx.lc : nx.rc;
                    if (f < 2 * NL && RECOMP && c < nl) continue;
                    const T *slab = f < 2 * NL ? V + vslot(c) * K * TC : B + (size_t)(nx.node - nl) * K * TC;
                    asm volatile("prefetch.global.L2 [%0];" :: "l"(slab + (f % NL) * (128 / sizeof(T))));
                }
            }
            for (int side = 0; side < 2; side++, sidx++) {
                const int c = side ? sn.rc : sn.lc;
                const int s = side ? sn.lc : sn.rc;
                const bool internal = c >= nl;
                const int buf = sidx & 1;
                int *eb_side = ebase + (npar ? 0 : buf * TC);
                if (side && npar) __syncthreads();     // the last side is finished with X, E^T and H
                if (internal) stage_rows<T, GR_THREADS>(Er, Pbase + (size_t)c * K2, tid);
                const T *Hg = reinterpret_cast<const T *>(a.Hmat) + ((size_t)rq.pset * a.nbr + c) * npar * K2;
                constexpr int NV = K2 * sizeof(T) / 16;
                if (npar) {
                    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Hb);
                    for (int f = tid; f < NV; f += GR_THREADS)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16 * f),
                                     "l"(reinterpret_cast<const char *>(Hg) + 16 * f) : "memory");
                    asm volatile("cp.async.commit_group;" ::: "memory");
                }
                // inter~ = beta~_p . v_s
                if (!RECOMP || s >= nl) {
                    const T *Vs = V + vslot(s) * K * TC;
                    for (int f = 4 * tid; f < K * TC; f += 4 * GR_THREADS) {
                        T bq[4], vq[4], x[4];
                        Vec4<T>::load(Bp + f, bq);
                        Vec4<T>::load(Vs + f, vq);
#pragma unroll
                        for (int i = 0; i < 4; i++) x[i] = bq[i] * vq[i];
                        ColStore<T, 4>::store(X + f, x);
                        if (npar) {
#pragma unroll
                            for (int i = 0; i < 4; i++) x[i] = x[i] * isT[f / TC];
                            ColStore<T, 4>::store(Q1 + f, x);
                        }
                    }
                } else {
                    for (int f = tid; f < K * TC; f += GR_THREADS) {
                        const T x = Bp[f] * leaf_part(Pbase, s, f / TC, f % TC);
                        X[f] = x;
                        if (npar) Q1[f] = x * isT[f / TC];
                    }
                }
                if (npar && internal) {
                    const T *Ac = Ascr + (size_t)(c - nl) * K * TC;
                    for (int f = 4 * tid; f < K * TC; f += 4 * GR_THREADS) {
                        T x[4];
                        Vec4<T>::load(Ac + f, x);
#pragma unroll
                        for (int i = 0; i < 4; i++) x[i] = x[i] * sqT[f / TC];
                        ColStore<T, 4>::store(Q2 + f, x);
                    }
                }
                if (tid < TC) {
                    const int eb = fS[(size_t)p * TC + tid] + e_of(s, tid);
                    eb_side[tid] = eb;
                    const int ex = eb + e_of(c, tid) - eroot[tid];
                    const bool far = ex <= -900 || ex >= 900;
                    wcol[buf * TC + tid] = far ? zt[tid] : zt[tid] * __hiloint2double((ex + 1023) << 20, 0);
                    wexp[buf * TC + tid] = far ? ex : 0;
                }
                // the child's own partial, for the gradient
                T vc[4][CPT];
                if (!RECOMP || internal) {
#pragma unroll
                    for (int i = 0; i < 4; i++) ColLoad<T, CPT>::load(V + (vslot(c) * K + a0 + i) * TC + c0, vc[i]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int cc = 0; cc < CPT; cc++) vc[i][cc] = leaf_part(Pbase, c, a0 + i, c0 + cc);
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                // gradient: (Q^T inter) . v_c per column, summed over this thread's 4 states
                T *rd = red + (size_t)buf * (1 + npar) * 16 * TC + ty * TC + c0;
                {
                    T wq[4][CPT];
                    contract<T, TC, KAHAN, CPT, GR_UNROLL>(Qs, X, a0, c0, wq);
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        T acc = (T)0;
#pragma unroll
                        for (int i = 0; i < 4; i++) acc += wq[i][cc] * vc[i][cc];
                        rd[cc] = acc;
                    }
                }
                flush();       // the last side's sums
                MU *cm = colmax + buf * TC, *cm_next = colmax + (buf ^ 1) * TC;
                T bt[4][CPT];
                if (internal) {
                    contract_rows<T, TC, KAHAN, GR_UNROLL>(Er, X, a0, c0, bt);
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        T mx = (T)0;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            bt[i][cc] += X[(a0 + i) * TC + c0 + cc];
                            mx = bt[i][cc] > mx ? bt[i][cc] : mx;
                        }
                        AtomMax<T>::upd(cm + c0 + cc, mx);
                    }
                }
                // parameters: inter^T (dP_c / dx) alpha_c = p^T H_x q with p = U^T D^-1/2 inter and
                // q = U^T D^1/2 alpha_c, for a leaf one row of U (its alpha_c is one-hot)
                T pv[4][CPT], qv[4][CPT];
                if (npar) {
                    contract<T, TC, KAHAN, CPT, GR_UNROLL>(Us, Q1, a0, c0, pv);
                    if (internal) {
                        contract<T, TC, KAHAN, CPT, GR_UNROLL>(Us, Q2, a0, c0, qv);
                    } else {
#pragma unroll
                        for (int cc = 0; cc < CPT; cc++) {
                            const int sl = lvT[c * TC + c0 + cc];
                            T u[4];
                            Vec4<T>::load(sl < K ? Us + sl * K + a0 : wmT + a0, u);
#pragma unroll
                            for (int i = 0; i < 4; i++) qv[i][cc] = sl < K ? u[i] * sqT[sl] : u[i];
                        }
                    }
                }
                __syncthreads();
                if (tid < TC) cm_next[tid] = 0;
                if (internal) {
                    T *Bc = B + (size_t)(c - nl) * K * TC;
                    int ecol[CPT];
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        const T mx = AtomMax<T>::get(cm + c0 + cc);
                        ecol[cc] = (mx > (T)0) ? exp_of(mx) : 0;
                        if (ty == 0) fS[(size_t)c * TC + c0 + cc] = eb_side[c0 + cc] + ecol[cc];
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        T y[CPT];
#pragma unroll
                        for (int cc = 0; cc < CPT; cc++) y[cc] = scale2(bt[i][cc], -ecol[cc]);
                        ColStore<T, CPT>::store(Bc + (size_t)(a0 + i) * TC + c0, y);
                    }
                }
                if (npar) {
                    // H_1 takes the place of E^T while H_0 is used; q takes that of D^-1/2 inter
                    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Er);
                    for (int f = tid; f < NV; f += GR_THREADS)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16 * f),
                                     "l"(reinterpret_cast<const char *>(Hg + K2) + 16 * f) : "memory");
                    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 4; i++) ColStore<T, CPT>::store(Q1 + (a0 + i) * TC + c0, qv[i]);
                    for (int x = 0; x < 2; x++) {
                        if (x) asm volatile("cp.async.wait_all;" ::: "memory");
                        __syncthreads();
                        T rv[4][CPT];
                        contract<T, TC, KAHAN, CPT, GR_UNROLL>(x ? Er : Hb, Q1, a0, c0, rv);
#pragma unroll
                        for (int cc = 0; cc < CPT; cc++) {
                            T acc = (T)0;
#pragma unroll
                            for (int i = 0; i < 4; i++) acc += pv[i][cc] * rv[i][cc];
                            rd[(size_t)(1 + x) * 16 * TC + cc] = acc;
                        }
                    }
                }
                pc = c;
                pb = buf;
            }
        }
        for (int k = 0; k < 2; k++) {      // the last two sides'
            __syncthreads();
            flush();
        }
        if (lane == 0 && warp >= 1 && warp <= npar) gout[a.nbr + warp - 1] = pacc;
    }
}

// The most shared memory a tree may ask for: three matrices, the slots and a tile of 64 (FP64: 32)
// columns, with the rate parameters U and two tiles more.  The kernel's own layout is smaller; the
// limit on trees is part of the interface.
size_t grad_smem_bytes(int prec, int nslots, int nl, int nint, int npar)
{
    const size_t es = prec == PCSF_PREC_FP64 ? 8 : 4, tc = prec == PCSF_PREC_FP64 ? 32 : 64;
    size_t b = es * (3 * (size_t)K2 + (size_t)nslots * K * tc + (size_t)K * tc + 16 * tc) + es * tc + 16 * tc +
               sizeof(SchedNode) * nint;
    b = (b + 15) & ~size_t(15);
    b = (b + (size_t)nl * tc + 15) & ~size_t(15);
    return b + (npar ? es * ((size_t)K2 + (nslots >= 2 ? 0 : 2 * (size_t)K * tc)) : 0);
}

int grad_tile_cols() { return GR_TC; }

template <typename T, int KAHAN, bool RECOMP>
static int ctas_per_sm_r(int nslots, int nl, int nint, int npar)
{
    const size_t smem = GradLayout<T, RECOMP>::smem(nslots, nl, nint, npar);
    int n = 0;
    if (allow_smem<k_grad<T, KAHAN, RECOMP>>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_grad<T, KAHAN, RECOMP>, GR_THREADS, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return std::max(n, 1);
}

int grad_ctas_per_sm(int prec, int nslots, int nl, int nint, int npar)
{
    if (prec == PCSF_PREC_FP64) return ctas_per_sm_r<double, 0, false>(nslots, nl, nint, npar);
    return ctas_per_sm_r<float, 2, false>(nslots, nl, nint, npar);
}

size_t grad_scratch_per_cta(int prec, int nl, int npar, bool recompute_leaves)
{
    if (prec == PCSF_PREC_FP64)
        return recompute_leaves ? GradLayout<double, true>::scratch(nl, npar) : GradLayout<double, false>::scratch(nl, npar);
    return recompute_leaves ? GradLayout<float, true>::scratch(nl, npar) : GradLayout<float, false>::scratch(nl, npar);
}

template <typename T, int KAHAN, bool RECOMP>
static cudaError_t launch_grad_r(const GradArgs &a, cudaStream_t s, int grid)
{
    size_t smem = GradLayout<T, RECOMP>::smem(a.nslots, a.nl, a.n_internal, a.npar);
    cudaError_t e = allow_smem<k_grad<T, KAHAN, RECOMP>>();
    if (e != cudaSuccess) return e;
    k_grad<T, KAHAN, RECOMP><<<grid, GR_THREADS, smem, s>>>(a);
    return cudaGetLastError();
}

template <typename T, int KAHAN>
static cudaError_t launch_grad_t(const GradArgs &a, cudaStream_t s, int grid)
{
    return a.recompute_leaves ? launch_grad_r<T, KAHAN, true>(a, s, grid) : launch_grad_r<T, KAHAN, false>(a, s, grid);
}

cudaError_t launch_grad(int prec, int comp, const GradArgs &a, cudaStream_t s, int grid)
{
    if (a.nwi <= 0) return cudaSuccess;
    if (prec == PCSF_PREC_FP64) return launch_grad_t<double, 0>(a, s, grid);
    if (comp == 1) return launch_grad_t<float, 1>(a, s, grid);
    if (comp == 2) return launch_grad_t<float, 2>(a, s, grid);
    return launch_grad_t<float, 0>(a, s, grid);
}

// H_x^T = (F(t) o Bdot_x)^T per (P set, branch, parameter).  F_ij = (e^{lam_i t} -
// e^{lam_j t}) / (lam_i - lam_j), written as e^{lam_j t} (e^{d t} - 1) / d with
// d = lam_i - lam_j and a Taylor series in d t when |d t| < 1e-2 (no cancellation).
// F is symmetric: a CTA takes HF_BRANCHES branches of a P set, its threads the 2,016 pairs i < j
// (1 / d and Bdot kept over the branches), F goes through shared memory and H out in rows.  The
// quotient is corrected to the division's rounding (q = x r, q + (x - q d) r; Markstein 1990).
// What bounds it: FP64 issue (two lanes per clock), about 14 instructions an entry where every
// entry formed its own quotient or series and wrote with a stride of a row; 40 P sets of 198
// branches 2.2 -> 0.75 ms.
constexpr int HF_BRANCHES = 16, HF_LD = K + 1;
template <typename T>
__global__ void __launch_bounds__(256) k_hform(const PSet *ps, const double *branch, int nbr, const double *lam,
                                               const T *Bdot, T *H)
{
    __shared__ double el[HF_BRANCHES][K];
    __shared__ double F[K * HF_LD];
    constexpr int NP = K * (K - 1) / 2, PER = (NP + 255) / 256;
    const int b0 = blockIdx.x * HF_BRANCHES, b1 = min(nbr, b0 + HF_BRANCHES), r = blockIdx.y, tid = threadIdx.x;
    const PSet rq = ps[r];
    const int md = rq.model;
    const double *lm = lam + (size_t)md * K;
    for (int f = tid; f < (b1 - b0) * K; f += 256) el[f / K][f % K] = exp(lm[f % K] * (rq.rho * branch[b0 + f / K]));
    int ij[PER];                 // the thread's pairs, row p / 64 of a 32 x 63 fold of the triangle
    double d[PER], rd[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int p = min(tid + 256 * k, NP - 1), i0 = p / (K - 1), j0 = p % (K - 1);
        // fold: row i0 holds (i0, j) for j > i0, then row K - 1 - i0's pairs
        const bool own = j0 >= i0;
        const int i = own ? i0 : K - 1 - i0, j = own ? j0 + 1 : K - 1 - j0;
        ij[k] = i << 8 | j;
        d[k] = lm[i] - lm[j];
        rd[k] = 1.0 / d[k];
    }
    double bd[2][K2 / 256];      // Bdot_x^T of the elements that the thread writes
#pragma unroll
    for (int k = 0; k < K2 / 256; k++)
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const int o = tid + 256 * k;
            bd[x][k] = (double)Bdot[((size_t)md * 2 + x) * K2 + (o % K) * K + o / K];
        }
    for (int b = b0; b < b1; b++) {
        const double t = rq.rho * branch[b];
        const double *e = el[b - b0];
        __syncthreads();         // el ready; the last branch's F is read
        if (tid < K) F[tid * HF_LD + tid] = t * e[tid];
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int i = ij[k] >> 8, j = ij[k] & 255;
            const double dt = d[k] * t;
            double v;
            if (fabs(dt) < 1e-2) {
                v = t * e[j] * (1.0 + dt * (0.5 + dt * (1.0 / 6.0 + dt * (1.0 / 24.0 + dt * (1.0 / 120.0)))));
            } else {
                const double x = e[i] - e[j], q = x * rd[k];
                v = fma(fma(-q, d[k], x), rd[k], q);
            }
            F[i * HF_LD + j] = v;
            F[j * HF_LD + i] = v;
        }
        __syncthreads();
        T *out = H + ((size_t)r * nbr + b) * 2 * K2;
#pragma unroll
        for (int k = 0; k < K2 / 256; k++) {
            const int o = tid + 256 * k;
            const double v = F[(o / K) * HF_LD + o % K];
            out[o] = (T)(v * bd[0][k]);
            out[K2 + o] = (T)(v * bd[1][k]);
        }
    }
}

cudaError_t launch_hform(bool fp64, const PSet *ps, int nps, const double *branch, int nbr, const double *lam,
                         const void *Bdot, void *H, cudaStream_t s)
{
    if (nps <= 0) return cudaSuccess;
    dim3 grid((nbr + HF_BRANCHES - 1) / HF_BRANCHES, nps);
    if (fp64) k_hform<double><<<grid, 256, 0, s>>>(ps, branch, nbr, lam, (const double *)Bdot, (double *)H);
    else k_hform<float><<<grid, 256, 0, s>>>(ps, branch, nbr, lam, (const float *)Bdot, (float *)H);
    return cudaGetLastError();
}

// grad[r][c] = sum of gpart over request r's work items (fixed order)
__global__ void k_reduce_grad(const double *gpart, const int32_t *wi_begin, int nreq, int nbr, double *grad)
{
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nreq * nbr) return;
    int r = idx / nbr, c = idx % nbr;
    double g = 0.0;
    for (size_t w = wi_begin[r]; w < (size_t)wi_begin[r + 1]; w++) g += gpart[w * nbr + c];
    grad[idx] = g;
}

cudaError_t launch_reduce_grad(const double *gpart, const int32_t *wi_begin, int nreq, int nbr, double *grad,
                               cudaStream_t s)
{
    if (nreq <= 0) return cudaSuccess;
    int tot = nreq * nbr;
    k_reduce_grad<<<(tot + 255) / 256, 256, 0, s>>>(gpart, wi_begin, nreq, nbr, grad);
    return cudaGetLastError();
}

// OmegaModel rate matrices and their derivatives in the eigenbasis, per model (its parameters
// key[m] = kappa, omega, sigma, F3x4) and parameter x = kappa, omega: Q (lib OmegaModel.ml:21-80,
// scaled to mean rate 1) and Bdot_x = U^T D^1/2 (dQ/dx) D^-1/2 U.  With R the unscaled matrix and
// s = -sum_i pi_i R_ii, Q = R / s and dQ/dx = R'/s - R s'/s^2 (pi does not depend on kappa or omega).
// One CTA per (model, x); two 64^3 products in FP64 (two lanes per clock on an SM: 120 us) are
// what bounds it.  On 16 host threads the matrices of 40 models took ~5 ms of a call.
constexpr int OD_THREADS = 256;

__device__ __forceinline__ int codon_nuc(int i, int pos) { return (i >> (4 - 2 * pos)) & 3; }

template <typename T>
__global__ void __launch_bounds__(OD_THREADS) k_omega_deriv(const double *keys, const double *U_all, const double *sq_all,
                                                            const double *isq_all, T *Qout, T *Bout)
{
    extern __shared__ __align__(16) unsigned char odsm[];
    double *A = reinterpret_cast<double *>(odsm);      // [K][K] D^1/2 dQ D^-1/2
    double *Us = A + K2;                                // [K][K]
    double *T1 = Us + K2;                               // [K][K] A U
    __shared__ double pi[K], rs[K], drs[K];
    __shared__ double tot_s[2];
    const int m = blockIdx.x, x = blockIdx.y, tid = threadIdx.x;
    const double *q = keys + 12 * (size_t)m;
    const double *U = U_all + (size_t)m * K2, *sq = sq_all + (size_t)m * K, *isq = isq_all + (size_t)m * K;
    auto sc = [&](int i) {
        double out = 1.0;
        for (int pos = 0; pos < 3; pos++) {
            const int n = codon_nuc(i, pos), base = 3 + 3 * pos;
            out *= ((n == 3) ? 1.0 : q[base + n]) / (q[base] + (q[base + 1] + (q[base + 2] + 1.0)));
        }
        return out;
    };
    if (tid < K) pi[tid] = sc(tid) / (1.0 - (1.0 - q[2]) * (sc(48) + (sc(50) + sc(56))));
    for (int f = tid; f < K2; f += OD_THREADS) Us[f] = U[f];
    __syncthreads();
    // R_ij and dR_ij / dx (i != j)
    const char *aa = "KNKNTTTTRSRSIIMIQHQHPPPPRRRRLLLLEDEDAAAAGGGGVVVV*Y*YSSSS*CWCLFLF";
    auto rate = [&](int i, int j, double &v, double &dv) {
        v = dv = 0.0;
        int nd = 0, a = 0, b = 0;
        for (int pos = 0; pos < 3; pos++)
            if (codon_nuc(i, pos) != codon_nuc(j, pos)) { nd++; a = codon_nuc(i, pos); b = codon_nuc(j, pos); }
        if (nd != 1) return;
        const bool transition = a + b == 2 ? a != 1 : a + b == 4 && a != 2;
        const bool nonsyn = aa[i] != '*' && aa[j] != '*' && aa[i] != aa[j];
        v = pi[j] * ((transition ? q[0] : 1.0) * (nonsyn ? q[1] : 1.0));
        if (x == 0 ? transition : nonsyn) dv = v / q[x];
    };
    if (tid < K) {
        double t = 0.0, dt = 0.0;
        for (int j = 0; j < K; j++) {
            double v, dv;
            rate(tid, j, v, dv);
            t += v;
            dt += dv;
        }
        rs[tid] = t;
        drs[tid] = dt;
    }
    __syncthreads();
    if (tid == 0) {
        double s = 0.0, ds = 0.0;
        for (int i = 0; i < K; i++) {
            s += pi[i] * rs[i];
            ds += pi[i] * drs[i];
        }
        tot_s[0] = s;
        tot_s[1] = ds;
    }
    __syncthreads();
    const double s = tot_s[0], ds = tot_s[1];
    for (int f = tid; f < K2; f += OD_THREADS) {
        const int i = f / K, j = f % K;
        double v, dv;
        rate(i, j, v, dv);
        if (i == j) {
            v = -rs[i];
            dv = -drs[i];
        }
        if (x == 0) Qout[(size_t)m * K2 + f] = (T)(v / s);
        A[f] = sq[i] * (dv / s - v * ds / (s * s)) * isq[j];
    }
    __syncthreads();
    // T1 = A U, Bdot = U^T T1: four rows and four columns per thread
    const int r0 = 4 * (tid / 16), c0 = 4 * (tid % 16);
    for (int pass = 0; pass < 2; pass++) {
        const double *L = pass ? Us : A, *M = pass ? T1 : Us;
        double acc[4][4] = {};
        for (int k = 0; k < K; k++) {
            double l[4], c[4];
#pragma unroll
            for (int i = 0; i < 4; i++) l[i] = pass ? L[k * K + r0 + i] : L[(r0 + i) * K + k];
            Vec4<double>::load(M + k * K + c0, c);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fma(l[i], c[j], acc[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (pass) Bout[((size_t)m * 2 + x) * K2 + (r0 + i) * K + c0 + j] = (T)acc[i][j];
                else T1[(r0 + i) * K + c0 + j] = acc[i][j];
            }
        __syncthreads();
    }
}

cudaError_t launch_omega_deriv(bool fp64, const double *keys, const double *U, const double *sq, const double *isq, int nmodels,
                               void *Q, void *Bdot, cudaStream_t s)
{
    if (nmodels <= 0) return cudaSuccess;
    const size_t smem = sizeof(double) * 3 * K2;
    const dim3 grid(nmodels, 2);
    cudaError_t e = fp64 ? allow_smem<k_omega_deriv<double>>()
                         : allow_smem<k_omega_deriv<float>>();
    if (e != cudaSuccess) return e;
    if (fp64) k_omega_deriv<double><<<grid, OD_THREADS, smem, s>>>(keys, U, sq, isq, (double *)Q, (double *)Bdot);
    else k_omega_deriv<float><<<grid, OD_THREADS, smem, s>>>(keys, U, sq, isq, (float *)Q, (float *)Bdot);
    return cudaGetLastError();
}

// Codons of each region's leaves, counted (codes above 63 are not): hist [nreg][64].  One CTA per
// region, a histogram per warp.
__global__ void __launch_bounds__(256) k_codon_hist(const uint8_t *codes, const int64_t *offs, int nl, unsigned long long *hist)
{
    __shared__ uint32_t h[8][K];
    const int r = blockIdx.x, tid = threadIdx.x;
    for (int f = tid; f < 8 * K; f += 256) h[f / K][f % K] = 0;
    __syncthreads();
    const size_t b1 = (size_t)offs[r + 1] * nl;
    for (size_t b = (size_t)offs[r] * nl + tid; b < b1; b += 256) {
        const int c = codes[b];
        if (c < K) atomicAdd(&h[tid >> 5][c], 1u);
    }
    __syncthreads();
    if (tid < K) {
        unsigned long long n = 0;
        for (int w = 0; w < 8; w++) n += h[w][tid];
        hist[(size_t)r * K + tid] = n;
    }
}

cudaError_t launch_codon_hist(const uint8_t *codes, const int64_t *offs, int nreg, int nl, unsigned long long *hist, cudaStream_t s)
{
    if (nreg <= 0) return cudaSuccess;
    k_codon_hist<<<nreg, 256, 0, s>>>(codes, offs, nl, hist);
    return cudaGetLastError();
}

}  // namespace pcsf
