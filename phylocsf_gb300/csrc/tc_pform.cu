// Tensor-core P(t) formation for the search evaluations of the tensor-core
// engines (FP32 grid correction, see k_pform in kernels.cu):
//
//   E(t) = E(t_g) + C,   C[i][j] = sum_m isq_i U_im cf_m U_jm sq_j,
//   cf_m = e^{lam_m t_g} expm1(lam_m (t - t_g)),
//
// where C, at most 0.1 % of E, is the only arithmetic that needs a GEMM.  Two
// branches of one P set form one M = 128 tile (rows 64 b + i): A[row][m] =
// isq_i U_im cf_m (staged per pair, TF32 hi / lo), B[j][m] = U_jm sq_j (fixed
// per model, pre-split on the host and fetched once per CTA by bulk copy), and
// D = A_lo B_hi + A_hi B_lo + A_hi B_hi in tensor memory (kind::tf32, N = 64,
// K = 64).  Thread r owns row r: the epilogue adds E(t_g) (or forms the
// below-grid Taylor E = tQ + t^2 Q^2 / 2), applies the clamp / renormalise row
// rule of Q.ml:226-247 with the diagonal as the compensated sum of the row, and
// writes what the tensor-core pruning kernel reads: E^T for the branches above
// leaves (row gathers) and the pre-split B operand for the branches above
// internal nodes.
//
// One CTA (128 threads) walks the branch pairs of one P set, or a part of them when the
// launch has few P sets (launch_pform_tc).  A_hi sits in tensor
// memory (columns 64..127, lane r = row r) and only A_lo in shared memory, so a CTA
// takes 64 KB of shared memory and 128 tensor-memory columns and three CTAs share an
// SM.  mbarrier waits are bounded as in the pruning kernel; on timeout the CTA records an
// error, waits (bounded) for its MMAs, frees its tensor memory and stops.
//
// What bounds it: the latency of its per-pair chain, 13,300 clocks beside two other CTAs
// (19,200 before): the rows of E(t_g) from L2 while the MMAs run 3,500, A 2,700 (4,900 when
// each lane read its own row of U: 32 lines an instruction; the host lays isq U out for
// coalesced reads now), the row's compensated sum 2,500 (3,800 with selects in its chain
// and a second pass to insert the diagonal), 1,600 of MMA issue, the row-sum check 850
// (1,900 with its operands looked up for every pair), and the next pair's coefficients
// formed in the MMAs' shadow.  Issue slots are a third used, HBM writes 30 %.  Measured, all
// P(t) launches of a call: 384 regions on 58 leaves 13.7 -> 11.0 ms, 60 genes on 100 leaves
// 8.1 -> 7.3 ms, ORF sets 1.42 -> 1.13 ms.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "pcsf_internal.h"
#include "prune_common.cuh"
#include "tc_common.cuh"

namespace pcsf {

constexpr int PFT_THREADS = 128;
constexpr uint32_t PFT_B = 0;          // [hi, lo][64 x 64]   B = U^T D^1/2, 2 x 16 KB
constexpr uint32_t PFT_A = 32768;      // [128 x 64]  A_lo, 32 KB
constexpr uint32_t PFT_SMEM = 65536;
constexpr uint32_t PFT_TMEM_COLS = 128;   // D in 0..63, A_hi in 64..127
constexpr int PFT_MAX_BRANCHES = 320;
constexpr int PFT_TARGET = 4 * 3;      // CTAs of a launch per SM: four waves of three

// diag -= x by Kahan's summation except where j == i, with the low part in dc: the last two of four
// additions are predicated, so nothing but them is on the chain
__device__ __forceinline__ void kahan_minus(float &diag, float &dc, float x, int i, int j)
{
    asm("{\n .reg .pred p;\n .reg .f32 y, s, t;\n setp.ne.s32 p, %3, %4;\n sub.rn.f32 y, %2, %1;\n"
        " add.rn.f32 s, %0, y;\n sub.rn.f32 t, s, %0;\n @p sub.rn.f32 %1, t, y;\n @p mov.f32 %0, s;\n}\n"
        : "+f"(diag), "+f"(dc) : "f"(-x), "r"(i), "r"(j));
}

__global__ void __launch_bounds__(PFT_THREADS, 3) k_pform_tc(const PSet *ps, const double *branch, int nbr, int nl,
                                                          DevModels m, const float *Bpf, float *Pbuf, float *Bop,
                                                          int32_t *status_key, int *err, int per_cta, int leaf_rows)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint32_t tbase_s;
    __shared__ __align__(8) uint64_t bar_mma, bar_b;
    __shared__ float cfs[2][2][K];      // [pair parity][branch of the pair]
    __shared__ double exs[2][2][K];     // expm1(lam_m t) where w_m != 0 (row-sum check)
    __shared__ int mode_g[PFT_MAX_BRANCHES];      // per branch: grid point << 2 | mode
    __shared__ float t_b[PFT_MAX_BRANCHES];       // t (FP32: the Taylor branch and expm1f only)
    __shared__ float h_b[PFT_MAX_BRANCHES];       // t - t_g, formed in FP64

    const int tid = threadIdx.x;
    const int r = blockIdx.x;           // P set (chunk-local)
    const int bb0 = blockIdx.y * per_cta, bb1 = min(nbr, bb0 + per_cta);   // this CTA's branches (bb0 even)
    const PSet rq = ps[r];
    const int md = rq.model;
    const uint32_t barM = smem_addr(&bar_mma), barB = smem_addr(&bar_b);
    const uint32_t sA = smem_addr(sm + PFT_A), sB = smem_addr(sm + PFT_B);
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
    const float4 *Uq = reinterpret_cast<const float4 *>(Bpf + 4 * K2 + (size_t)md * K2);   // [m / 4][i] isq_i U_im
    const double *lam = m.lam + md * K;
    const double *wrow = m.wrow + md * K;
    const int i = tid & (K - 1), bsel = tid >> 6;      // this thread's row: branch b0 + bsel, state i

    if ((tid >> 5) == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tbase_s)), "r"(PFT_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(barM), "r"(1));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(barB), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tbase_s;
    bool ok = true;
    if (tid == 0) {
        bulk_load(sB, Bpf + (size_t)md * 2 * K2, 2 * 16384, barB);
        ok = mbar_wait(barB, 0);
    }
    const uint32_t lane_off = (uint32_t)(((tid >> 5) & 3) * 32) << 16;
    uint32_t ph = 0;
    bool pending = false;               // an MMA group was issued and its completion not seen
    // per branch: 0 t = 0, 1 below the grid (Taylor), 2 grid correction at point g
    for (int b = bb0 + tid; b < bb1; b += PFT_THREADS) {
        const double t = rq.rho * branch[b];
        int mode = 0, g = 0;
        if (t == 0.0) mode = 0;
        else if (t < m.grid_t[0]) mode = 1;
        else {
            mode = 2;
            g = grid_point(m, t);
        }
        mode_g[b] = (g << 2) | mode;
        t_b[b] = (float)t;
        h_b[b] = (mode == 2) ? (float)(t - m.grid_t[g]) : 0.0f;
    }
    // FP32 copies of this thread's eigenvalue and its stationary-direction flag
    // (FP64 runs at a small fraction of the FP32 rate on this part)
    const float lam_i = (float)lam[i];
    bool listed = false;
    {
        const int16_t *wl = m.wlist + md * WLIST;
        if (wl[0] == -2) listed = (wrow[i] != 0.0);
        else
            for (int k = 0; k < WLIST; k++) listed |= (wl[k] == i);
    }
    const float ntol = -(float)m.tol, dtol = (float)(-1.0 - m.tol);
    // the row-sum check's one term (rowsum_minus_one), where the model has just one
    const int w0 = m.wlist[md * WLIST];
    const bool one_w = w0 >= 0 && m.wlist[md * WLIST + 1] < 0;
    const double wu = one_w ? m.U[(size_t)md * K2 + (size_t)i * K + w0] : 0.0, ww = one_w ? wrow[w0] : 0.0;
    const double isq_i = m.isq[md * K + i];

    // the coefficients cf of a pair of branches: thread (bsel, i) supplies coefficient m = i
    auto coefficients = [&](int b0, int par) {
        const int b = b0 + bsel;
        const int mg = (b < bb1) ? mode_g[b] : 0;
        float cf = 0.0f;
        if ((mg & 3) == 2) cf = m.grid_eg[((size_t)md * m.grid_n + (mg >> 2)) * K + i] * expm1f(lam_i * h_b[b]);
        cfs[par][bsel][i] = cf;
        exs[par][bsel][i] = listed ? (double)expm1f(lam_i * (b < bb1 ? t_b[b] : 0.0f)) : 0.0;
    };
    __syncthreads();                                  // per-branch table ready
    coefficients(bb0, 0);

    for (int b0 = bb0, par = 0; b0 < bb1; b0 += 2, par ^= 1) {
        const int b = b0 + bsel;                      // this thread's branch
        if (__syncthreads_or(!ok)) break;             // coefficients ready / previous pair done
        const int mode = (b < bb1) ? (mode_g[b] & 3) : 0, g = (b < bb1) ? (mode_g[b] >> 2) : 0;
        const float t = (b < bb1) ? t_b[b] : 0.0f;
        // ---- A operand: row tid = isq_i U_im cf_m, TF32 hi (tensor memory) / lo (shared)
        {
            const float *cf = cfs[par][bsel];
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                float h[16];
#pragma unroll
                for (int q4 = 0; q4 < 4; q4++) {
                    const int q = 4 * c + q4;
                    const float4 u = __ldg(Uq + q * K + i);
                    const float x0 = u.x * cf[4 * q], x1 = u.y * cf[4 * q + 1];
                    const float x2 = u.z * cf[4 * q + 2], x3 = u.w * cf[4 * q + 3];
                    const float4 hv = make_float4(tf32_hi(x0), tf32_hi(x1), tf32_hi(x2), tf32_hi(x3));
                    *reinterpret_cast<float4 *>(sm + PFT_A + core_off(tid, 4 * q, 16)) =
                        make_float4(x0 - hv.x, x1 - hv.y, x2 - hv.z, x3 - hv.w);
                    h[4 * q4] = hv.x; h[4 * q4 + 1] = hv.y; h[4 * q4 + 2] = hv.z; h[4 * q4 + 3] = hv.w;
                }
                tmem_st16(tbase + lane_off + 64 + 16 * c, h);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (tid == 0) {
            mma3_tf32_ta(tbase, tbase + 64, sA, sB, 16384, idesc);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(barM) : "memory");
        }
        // ---- epilogue inputs that do not depend on D, loaded while the MMAs run (before A is formed
        // they cost more than they hide: A's own loads then wait behind them)
        float row[K];
        {
            const float *eg = m.gridT + ((size_t)md * m.grid_n + g) * K2;   // E(t_g)^T
            const float *Qf = m.Qf + (size_t)md * K2 + (size_t)i * K, *Q2f = m.Q2f + (size_t)md * K2 + (size_t)i * K;
            const float tt = t, h2 = 0.5f * t * t;
#pragma unroll
            for (int j = 0; j < K; j++) {
                if (mode == 2) row[j] = __ldg(eg + (size_t)j * K + i);
                else if (mode == 1) row[j] = tt * Qf[j] + h2 * Q2f[j];
                else row[j] = 0.0f;
            }
        }
        if (b0 + 2 < bb1) coefficients(b0 + 2, par ^ 1);      // the next pair's, while the MMAs run
        pending = true;
        const bool done = mbar_wait(barM, ph);
        ph ^= 1u;
        if (done) pending = false;
        tc_fence_after();
        if (mode == 2) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
                float d[16];
                tmem_ld16(tbase + lane_off + 16 * c, d);
#pragma unroll
                for (int j = 0; j < 16; j++) row[16 * c + j] += d[j];
            }
        }
        tc_fence_before();
        if (b < bb1 && done) {
            // branch-free in j: i differs per lane, and a branch on j == i would split the
            // warp into single-lane paths for everything that follows.  Off the diagonal:
            // diag -= x (Kahan), the step's last two operations predicated, so that its chain
            // is four additions; row[i] is not used any more (the diagonal is stored by itself)
            bool neg = false;
            float diag = 0.0f, dc = 0.0f;
#pragma unroll
            for (int j = 0; j < K; j++) {
                neg |= row[j] < (j == i ? dtol : ntol);
                row[j] = fmaxf(row[j], 0.0f);             // clamp an off-diagonal negative
                kahan_minus(diag, dc, row[j], i, j);
            }
            const double rs = one_w ? wu * exs[par][bsel][w0] * ww * isq_i : rowsum_minus_one(m, md, i, exs[par][bsel]);
            if (neg) status_min(status_key + r, b, i, PCSF_ENEGP);
            else if (fabs(rs) > m.tol) status_min(status_key + r, b, i, PCSF_EROWSUM);
            else if (!(diag > -1.0f)) status_min(status_key + r, b, i, PCSF_EDIAG);
            if (b >= nl) {      // above an internal node: the pruning kernel's B operand
                float *dst = Bop + ((size_t)r * (nbr - nl) + (b - nl)) * 2 * K2;
#pragma unroll
                for (int q = 0; q < K / 4; q++)
                    bop_store(dst, i, q, make_float4(row[4 * q], row[4 * q + 1], row[4 * q + 2], row[4 * q + 3]));
                dst += (i >> 2) * 256 + i * 4 + (i & 3);
                dst[0] = tf32_hi(diag);
                dst[K2] = diag - tf32_hi(diag);
            } else {            // above a leaf: E^T rows for the gathers, or k_prune_tc's P^T rows
                float *out = Pbuf + ((size_t)r * nbr + b) * K2 + (leaf_rows ? leaf_pos(i) - i : 0);
#pragma unroll
                for (int j = 0; j < K; j++) out[(size_t)j * K + i] = row[j];
                out[(size_t)i * K + i] = leaf_rows ? diag + 1.0f : diag;
            }
        }
        if (!done) ok = false;      // agreed on at the next pair's first barrier
        tc_fence_after();
    }
    if (__syncthreads_or(!ok)) ok = false;
    // bounded again: the first fetch and the last MMAs may still be on their way after a wait that ran out
    if (!ok && tid == 0) {
        atomicExch(err, 1);
        mbar_wait(barB, 0);
    }
    if (pending) mbar_wait(barM, ph ^ 1u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if ((tid >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(PFT_TMEM_COLS));
}

cudaError_t launch_pform_tc(const PSet *ps, int nps, const double *branch, int nbr, int nl, DevModels m,
                            const float *Bpf, float *Pbuf, float *Bop, int32_t *status_key, int *err, cudaStream_t s,
                            bool leaf_rows)
{
    if (nps <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_pform_tc, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) e = allow_smem<k_pform_tc>();
    if (e != cudaSuccess) return e;
    // Branch pairs per CTA: all of a P set's when there are enough P sets to fill the GPU
    // several times over, fewer for a short list (one exon's search round asks for two to six
    // P sets): about PFT_TARGET CTAs per SM in all, at the price of one 32 KB fetch of B per CTA.
    // Measured, P(t) of one mle call on 58 leaves: 1 region (2-6 P sets a round) 5.1 -> 0.28 ms,
    // 384 regions (~800 P sets a round: 1.7 waves before, three CTAs per P set now) 20.0 -> 14.6 ms,
    // both before the chain was shortened.
    const int pairs = (nbr + 1) / 2;
    const int want = std::min(pairs, std::max(1, (PFT_TARGET * m.sm_count + nps - 1) / nps));
    const int per_cta = 2 * ((pairs + want - 1) / want);
    const dim3 grid(nps, (nbr + per_cta - 1) / per_cta);
    k_pform_tc<<<grid, PFT_THREADS, PFT_SMEM, s>>>(ps, branch, nbr, nl, m, Bpf, Pbuf, Bop, status_key, err, per_cta,
                                                       leaf_rows ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace pcsf
