// Tensor-core (tcgen05, sm_103a) pruning kernel.
//
// Same contract as k_prune (kernels.cu) -- one work item is a tile of columns of
// one request's region, walked through the register-minimal schedule -- with the
// internal-branch contractions on the 5th-generation tensor cores:
//
//   D_c[site][a] = sum_j alpha_c[site][j] * E_c[a][j]      (M = 128 sites, N = 64, K = 64)
//
// as kind::tf32 MMAs with FP32 accumulation in tensor memory.  TF32 keeps 10
// mantissa bits, so each operand is split into hi = tf32(x) (the MMA ignores the
// low 13 bits) and lo = x - hi, and D = A_lo B_hi + A_hi B_lo + A_hi B_hi (the
// small products first), which restores ~22 bits.  The epilogue adds the exact
// identity part, v_c = alpha_c + D_c (E = P - I), so rounding in D only touches
// the off-diagonal mass of P.
//
// Layout: 256 threads, eight warps of 16 tile columns; four threads share a column.  A
// thread holds 16 states of two columns, as the 16x256b tensor-memory accesses hand them
// out (pairs of states 8 i + 2 (lane % 4), + 1), so a column's maximum is two shuffles away
// and no warp waits for another between a contraction and the next staging.  A node's
// normalised partial stays in those registers: the schedule evaluates a node's last
// internal child just before the node, so its partial goes from there into the
// contraction's operands (hi and lo, both in tensor memory) and is still there when D
// arrives.  Only the first of two internal children waits, on a stack whose top entry is in
// tensor memory (A hi, A lo, D, top: 256 columns) and the rest in global memory (L2).  With
// 66 KB of shared memory and 128 registers a thread two CTAs share an SM.
// B operands are pre-split by the P(t) kernel into the operand layout; one thread fetches
// each with a 32 KB bulk copy (cp.async.bulk, completion on an mbarrier), two contractions
// ahead.  One thread issues the MMAs when the eight warps have arrived on an mbarrier.
// Leaf children are gathers of P^T rows from L2 while the MMAs run: the P(t) kernel writes
// a leaf branch's rows with the identity added and the states permuted (leaf_pos) so that
// the four threads of a column read a row with 32-byte loads, each row's 256 bytes in two
// instructions of eight rows.  The root stage forms z = pi . alpha as an FP32 compensated
// dot product and log z = log m + e ln 2 (m in [0.5, 1)), with FP64 only for the per-column
// log and the tile sums.
//
// What bounds it: the latency of the per-node chain, about 5,000 clocks a node beside one
// other CTA: 24 MMAs of 60 clocks (N = 64 fills half of the tensor pipe's width, and a wider
// N would need the two halves of B in one MMA, another order of the sums), the staging
// and arrival before them (1,000) and the epilogue (800); a node with two leaves waits
// 1,700 for its rows.  Tensor pipe and issue slots are each about half used.  Registers
// decide: one more 32-byte array per thread spills, and spilling variants measured 10 to
// 40 % slower, so the rows are not fetched a node ahead.
// Measured, all search launches of a call: 384 regions on 58 leaves 46.5 -> 31.0 ms, 60 genes
// (106,356 columns) on 100 leaves 30.4 -> 20.3 ms, one region on 58 leaves (3 tiles a launch)
// 159 -> 122 us a launch.  Before, two threads owned a column (32 states each): every child's
// partial was stored and loaded again, a lane gathered its row alone (32 lines an
// instruction, a third of the LSU's wavefronts were leaf reads), and the maximum crossed
// warps through shared memory.
//
// Accuracy: the tensor cores' FP32 accumulation is not round-to-nearest: it
// rounds toward minus infinity (a measured mean of -5.7 ulp of the result over
// one K = 64 product, i.e. 8 accumulation steps, for positive and for negative
// results alike), so these values carry a small systematic error.  The engine
// therefore uses this kernel for the search evaluations of the rho maximisation
// and reports every returned likelihood from the compensated FP32 kernel.
//
// Every mbarrier wait is bounded; on timeout the kernel records an error, waits
// (again bounded) for its outstanding copies and tensor-core work, releases its
// tensor memory and exits.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "pcsf_internal.h"
#include "prune_common.cuh"
#include "tc_common.cuh"

namespace pcsf {

constexpr int TCP_THREADS = 256;     // eight warps of 16 tile columns
constexpr int TCP_M = 128;
constexpr int TCP_MAX_SLOTS = 8;
constexpr int TCP_MAX_LEAVES = 160;
// tensor memory: A hi, A lo, D, and the top of the stack, 64 columns each
constexpr uint32_t TCP_TMEM_COLS = 256, TM_HI = 0, TM_LO = 64, TM_D = 128, TM_S = 192;

// dynamic shared-memory map (bytes)
constexpr uint32_t SM_B = 0;            // two B operands, [hi, lo][64 x 64 fp32] = 2 x 16 KB each
constexpr uint32_t SM_SCHED = 65536;    // the schedule, contraction order, leaf states
constexpr uint32_t B_BYTES = 16384;
constexpr int LV_STRIDE = TCP_M;     // leaf-state rows: [leaf][site] bytes, words XOR-swizzled per row
// byte offset of (leaf l, site c): row l's 4-byte words are permuted by XOR with l mod 32,
// so that the fill (consecutive threads on consecutive leaves of one site) and the reads
// (consecutive threads on consecutive sites of one leaf) are both free of bank conflicts
__device__ __forceinline__ int lv_off(int l, int c) { return l * LV_STRIDE + (c ^ ((l & 31) << 2)); }

// the schedule as the kernel walks it: children (the leaf, if one is), what to do with them
struct TcNode {
    int16_t lc, rc;
    int32_t flags;
};
constexpr int TN_LEAVES = 1, TN_LEAF = 2;    // two leaves; one leaf (lc)
constexpr int TN_PUSH = 4;                   // the next node does not take the partial: it waits on the stack
static __host__ __device__ size_t tc_sched_bytes(int nint) { return ((size_t)nint * (sizeof(TcNode) + 2) + 15) & ~(size_t)15; }

__device__ const __align__(32) float ones_row[K] = {
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
    1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};

// four pairs of floats in one 256-bit load, pinned where it stands (before the wait that hides it)
__device__ __forceinline__ void ldg4(const float *p, f2 &a, f2 &b, f2 &c, f2 &d)
{
    float r[8];
    asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "l"(p));
    a = pk(r[0], r[1]); b = pk(r[2], r[3]); c = pk(r[4], r[5]); d = pk(r[6], r[7]);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count));
}
// one arrival for the warp: what its lanes did before is visible to those that wait
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane)
{
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
// stack entries below the one in tensor memory
static __host__ __device__ int prune_tc_levels(int depth) { return depth > 2 ? depth - 1 : 1; }

template <int NPROD>
__global__ void __launch_bounds__(TCP_THREADS, 2) k_prune_tc(PruneArgs a, float *stack, int *err)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint32_t tbase_s;
    __shared__ __align__(8) uint64_t bar_a, bar_mma, bar_b[2];
    __shared__ float zpart[2][2][TCP_M], prf[K], wlf[K];
    __shared__ int esc[TCP_M];
    __shared__ double red_l[TCP_M / 32], red_e[TCP_M / 32];
    __shared__ int nbseq_s, late_s;
    __shared__ struct { int w, k, ps, n, done; } ld;   // B loads: see load_next_b (kept by thread 32)

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nl = a.nl;
    TcNode *sched = reinterpret_cast<TcNode *>(sm + SM_SCHED);
    int16_t *bseq = reinterpret_cast<int16_t *>(sched + a.n_internal);   // internal child of each contraction, in order
    uint8_t *lvs = sm + SM_SCHED + tc_sched_bytes(a.n_internal);
    // operands staged (A), contraction done (M), B operand fetched (B)
    const uint32_t barA = smem_addr(&bar_a), barM = smem_addr(&bar_mma), barB = smem_addr(bar_b);
    const uint32_t sB = smem_addr(sm + SM_B);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tbase_s)), "r"(TCP_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        mbar_init(barA, TCP_THREADS / 32);
        mbar_init(barM, 1);
        mbar_init(barB, 1);
        mbar_init(barB + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int f = tid; f < a.n_internal; f += TCP_THREADS) {
        const SchedNode sn = a.sched[f], nx = a.sched[min(f + 1, a.n_internal - 1)];
        const bool ll = sn.lslot < 0, rl = sn.rslot < 0;
        TcNode t;
        t.lc = ll || !rl ? sn.lc : sn.rc;
        t.rc = ll || !rl ? sn.rc : sn.lc;
        t.flags = (ll && rl ? TN_LEAVES : ll || rl ? TN_LEAF : 0);
        if (f + 1 < a.n_internal && nx.lc != sn.node && nx.rc != sn.node) t.flags |= TN_PUSH;
        sched[f] = t;
    }
    if (tid == 0) {
        // contraction order: the child evaluated just before its parent, then the one that waits
        int k = 0, prev = -1;
        for (int f = 0; f < a.n_internal; f++) {
            const SchedNode sn = a.sched[f];
            const bool li = sn.lslot >= 0, ri = sn.rslot >= 0;
            if (li && ri) {
                bseq[k++] = prev == sn.lc ? sn.lc : sn.rc;
                bseq[k++] = prev == sn.lc ? sn.rc : sn.lc;
            } else if (li || ri) {
                bseq[k++] = li ? sn.lc : sn.rc;
            }
            prev = sn.node;
        }
        nbseq_s = k;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tbase_s;
    bool bad = false;       // a wait ran out: later waits are skipped, nothing more is issued
    int n = 0;              // contractions so far

    // B operands, two contractions ahead (thread 32).  ld: the next load's work item, index into bseq
    // and P set; loads issued, contractions done.
    auto load_next_b = [&]() {          // buffer ld.n % 2 is free
        const int nbseq = nbseq_s;
        if (ld.w >= a.nwi || nbseq == 0) return;
        const int c = bseq[ld.k], i = ld.n & 1;
        bulk_load(sB + i * 2 * B_BYTES, reinterpret_cast<const float *>(a.Bop) + ((size_t)ld.ps * a.nbop + (c - nl)) * 2 * K2,
                  2 * B_BYTES, barB + 8 * i);
        ld.n++;
        if (++ld.k == nbseq) {
            ld.k = 0;
            ld.w += gridDim.x;
            if (ld.w < a.nwi) ld.ps = a.req[a.wi[ld.w].request].pset;
        }
    };
    if (tid == 0) late_s = -1;
    if (tid == 32) {
        ld.w = blockIdx.x;
        ld.k = ld.n = ld.done = 0;
        ld.ps = (int)blockIdx.x < a.nwi ? a.req[a.wi[blockIdx.x].request].pset : 0;
        load_next_b();
        load_next_b();
    }

    // D = A_lo B_hi + A_hi B_lo + A_hi B_hi, once every warp has staged (warp 0, lane 0).
    // kind::tf32, D f32, A/B tf32, both K-major, N = 64, M = 128.  Descriptors advance in 16-byte
    // units: K-step 2048 B, lo half 16 KB, buffer 32 KB.
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t dB = sdesc(sB, 1024, 128);
    auto contract = [&]() {
        if (bad || !mbar_wait(barB + 8 * (n & 1), (n >> 1) & 1) || !mbar_wait(barA, n & 1)) {
            bad = true;
            return;
        }
        tc_fence_after();
        const uint64_t dBhi = dB + (uint64_t)(n & 1) * (2 * B_BYTES / 16), dBlo = dBhi + B_BYTES / 16;
        if (NPROD == 3) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                mma_tf32_ta(tbase + TM_D, tbase + TM_LO + 8 * j, dBhi + 128 * j, idesc, j > 0);
                mma_tf32_ta(tbase + TM_D, tbase + TM_HI + 8 * j, dBlo + 128 * j, idesc, 1);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            mma_tf32_ta(tbase + TM_D, tbase + TM_HI + 8 * j, dBhi + 128 * j, idesc, NPROD == 3 || j > 0);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(barM) : "memory");
    };

    // a partial of the thread's two columns is v[16]: pair i of column k (states 8 i + 2 (lane % 4),
    // + 1) at 2 i + k
    const int c0 = 32 * (warp & 3) + 16 * (warp >> 2);      // the warp's first column (TMEM lane)
    const uint32_t trow = tbase + ((uint32_t)c0 << 16);
    float *stk = stack + (size_t)blockIdx.x * prune_tc_levels(a.depth) * (32 * TCP_THREADS) + 2 * tid;

    // a partial into the A operand, hi and lo
    auto stage = [&](const f2 *x) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            f2 h[8], l[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float y, z;
                upk(x[8 * q + j], y, z);
                h[j] = pk(tf32_hi(y), tf32_hi(z));
                l[j] = sub2(x[8 * q + j], h[j]);
            }
            tmem_st_rows(trow + TM_HI + 32 * q, h);
            if (NPROD == 3) tmem_st_rows(trow + TM_LO + 32 * q, l);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        warp_arrive(barA, lane);
    };
    auto issue = [&]() {
        if (warp == 0) {
            if (lane == 0) contract();
            __syncwarp();
        }
    };
    auto wait_d = [&]() {
        if (!bad && !mbar_wait(barM, n & 1)) {
            bad = true;
            if (tid == 0) late_s = n & 1;       // its commit may still arrive
        }
        n++;
        __syncwarp();
        tc_fence_after();
        if (tid == 32 && !bad) {
            ld.done++;
            load_next_b();      // the B operand is free again
        }
    };

    for (int w = blockIdx.x; w < a.nwi; w += gridDim.x) {
        const WorkItem wi = a.wi[w];
        const Request rq = a.req[wi.request];
        const int md = rq.model;
        const float *Pbase = reinterpret_cast<const float *>(a.Pbuf) + (size_t)rq.pset * a.nbr * K2;
        const int ncols = wi.ncols;
        // the warp's leaf states (K: missing, and columns past the end)
        {
            const uint8_t *lg = a.leaves + ((size_t)wi.col0 + c0) * nl;
            const int nf = max(min(ncols - c0, 16), 0) * nl;
            __syncwarp();
            for (int f0 = 0; f0 < 16 * nl; f0 += 32 * 16) {
                uint8_t x[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int f = f0 + 32 * i + lane;
                    x[i] = f < nf ? __ldg(lg + f) : (uint8_t)K;
                }
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int f = f0 + 32 * i + lane, c = f / nl;
                    if (f < 16 * nl) lvs[lv_off(f - c * nl, c0 + c)] = x[i];
                }
            }
            __syncwarp();
        }
        // rows of a leaf's P^T (ones where it is missing) for the thread's two columns
        auto leaf_rows = [&](int l, f2 *x) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int s = lvs[lv_off(l, c0 + 8 * k + (lane >> 2))];
                const float *p = (s < K ? Pbase + (size_t)l * K2 + s * K : ones_row) + 8 * (lane & 3);
                ldg4(p, x[k], x[2 + k], x[4 + k], x[6 + k]);
                ldg4(p + 32, x[8 + k], x[10 + k], x[12 + k], x[14 + k]);
            }
        };
        int escale[2] = {0, 0};     // the columns' sums of rescale exponents
        int sp = 0;                 // stack entries in use
        f2 v[16];                   // a node's partial under construction, then normalised
        TcNode sn = sched[0];

#pragma unroll 1
        for (int ni = 0; ni < a.n_internal; ni++) {
            const int fl = sn.flags;
            f2 x[16];
            if (fl & TN_LEAVES) {
                leaf_rows(sn.lc, v);
                leaf_rows(sn.rc, x);
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = mul2(v[j], x[j]);
            } else {
                // the last node's partial (in v) is contracted first
                stage(v);
                if (fl & TN_LEAF) {
                    issue();
                    leaf_rows(sn.lc, x);
                } else if (--sp == 0) {
                    tmem_ld_rows(trow + TM_S, x);
                    tmem_ld_rows(trow + TM_S + 32, x + 8);
                } else {
                    const f2 *e = reinterpret_cast<const f2 *>(stk + (size_t)(sp - 1) * (32 * TCP_THREADS));
#pragma unroll
                    for (int j = 0; j < 16; j++) x[j] = e[j * TCP_THREADS];
                }
                if (!(fl & TN_LEAF)) issue();
                wait_d();
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    f2 d[8];
                    tmem_ld_rows(trow + TM_D + 32 * q, d);
#pragma unroll
                    for (int j = 0; j < 8; j++) v[8 * q + j] = add2(v[8 * q + j], d[j]);
                }
                if (fl & TN_LEAF) {
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = mul2(v[j], x[j]);
                } else {
                    // then the one from the stack
                    stage(x);
                    issue();
                    wait_d();
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        f2 d[8];
                        tmem_ld_rows(trow + TM_D + 32 * q, d);
#pragma unroll
                        for (int j = 0; j < 8; j++) v[8 * q + j] = mul2(v[8 * q + j], add2(x[8 * q + j], d[j]));
                    }
                }
            }
            sn = sched[min(ni + 1, a.n_internal - 1)];
            // ---- rescale each column by an exact power of two
            float mx[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    float y, z;
                    upk(v[2 * i + k], y, z);
                    m0 = fmaxf(m0, y);
                    m1 = fmaxf(m1, z);
                }
                mx[k] = fmaxf(m0, m1);
            }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
#pragma unroll
                for (int k = 0; k < 2; k++) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
            }
            // the biased exponents: a normal maximum below 2^126 scales with one multiplication
            const int b0 = __float_as_int(mx[0]) >> 23, b1 = __float_as_int(mx[1]) >> 23;
            if (__all_sync(0xffffffffu, min(b0, b1) > 0 && max(b0, b1) < 253)) {
                const float g0 = __int_as_float((253 - b0) << 23), g1 = __int_as_float((253 - b1) << 23);
                escale[0] += b0 - 126;
                escale[1] += b1 - 126;
                const f2 gg[2] = {pk(g0, g0), pk(g1, g1)};
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = mul2(v[j], gg[j & 1]);
            } else {
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const int e = mx[k] > 0.0f ? exp_of(mx[k]) : 0;
                    escale[k] += e;
                    const float h = scale2(1.0f, -(e >> 1)), l = scale2(1.0f, -(e - (e >> 1)));
#pragma unroll
                    for (int i = 0; i < 8; i++) v[2 * i + k] = mul2(mul2(v[2 * i + k], pk(h, h)), pk(l, l));
                }
            }
            if (fl & TN_PUSH) {
                if (sp == 0) {
                    tmem_st_rows(trow + TM_S, v);
                    tmem_st_rows(trow + TM_S + 32, v + 8);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                } else {
                    f2 *t = reinterpret_cast<f2 *>(stk + (size_t)(sp - 1) * (32 * TCP_THREADS));
#pragma unroll
                    for (int k = 0; k < 16; k++) t[k * TCP_THREADS] = v[k];
                }
                sp++;
            }
        }
        // ---- root, two threads per column: z = alpha_root . prior (FP32, compensated) and the
        // elpr term; log z = log m + e ln 2 with m in [0.5, 1) (logf of m is within ~4e-8
        // absolute, far below the tensor-core noise of these search values); FP64 only for the
        // per-column log and the sums over the tile (this part's FP64 rate is ~1/64 of FP32).
        // The partials change threads through the idle A operand.
        tmem_st_rows(trow + TM_HI, v);
        tmem_st_rows(trow + TM_HI + 32, v + 8);
        if ((lane & 3) == 0) {
            esc[c0 + (lane >> 2)] = escale[0];
            esc[c0 + 8 + (lane >> 2)] = escale[1];
        }
        if (tid < K) {
            prf[tid] = (float)a.m.prior[md * K + tid];
            wlf[tid] = (float)a.m.wlog[md * K + tid];
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        bad = __syncthreads_or(bad);
        if (bad) break;
        tc_fence_after();
        const int site = tid & (TCP_M - 1), half = tid >> 7, s0 = 32 * half;
        const int es = esc[site];
        {
            const uint32_t t = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + TM_HI + s0;
            float z = 0.0f, zc = 0.0f, wz = 0.0f;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                float u[16];
                tmem_ld16(t + 16 * q, u);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float y = u[j] * prf[s0 + 16 * q + j] - zc;
                    const float r = z + y;
                    zc = (r - z) - y;
                    z = r;
                    wz = fmaf(u[j], wlf[s0 + 16 * q + j], wz);
                }
            }
            zpart[half][0][site] = z;
            zpart[half][1][site] = wz;
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (half == 0) {
            double tl = 0.0, te = 0.0;
            if (site < ncols) {
                const float z = zpart[0][0][site] + zpart[1][0][site];
                const float wz = zpart[0][1][site] + zpart[1][1][site];
                if (z > 0.0f) {
                    int ez;
                    const float mz = frexpf(z, &ez);
                    tl = (double)logf(mz) + (double)(ez + es) * 0.69314718055994530942;
                    te = (double)(wz / z);
                } else {
                    tl = -INFINITY;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tl += __shfl_down_sync(0xffffffffu, tl, o);
                te += __shfl_down_sync(0xffffffffu, te, o);
            }
            if (lane == 0) { red_l[warp] = tl; red_e[warp] = te; }
            asm volatile("bar.sync 6, 128;" ::: "memory");
            if (tid == 0) {
                double sl = 0.0, se = 0.0;
                for (int k = 0; k < TCP_M / 32; k++) { sl += red_l[k]; se += red_e[k]; }
                a.partials[2 * (size_t)w] = sl;
                a.partials[2 * (size_t)w + 1] = se;
            }
        }
    }
    // quiesce: bulk copies may be outstanding, and after a timed-out wait for a contraction its
    // commit may still arrive; every wait is bounded
    if (tid == 32) {
        for (int i = ld.done; i < ld.n; i++) {
            if (!mbar_wait(barB + 8 * (i & 1), (i >> 1) & 1)) bad = true;
        }
    }
    if (tid == 0 && late_s >= 0) mbar_wait(barM, late_s);
    if (bad && lane == 0) atomicExch(err, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(TCP_TMEM_COLS));
}

bool prune_tc_supported(int nslots, int nl) { return nslots <= TCP_MAX_SLOTS && nl <= TCP_MAX_LEAVES; }

bool prune_tc_shape_ok(int shape) { return shape >= 0 && shape < PCSF_TC_SHAPES; }

size_t prune_tc_smem_bytes(int nl, int nint) { return SM_SCHED + tc_sched_bytes(nint) + (size_t)nl * LV_STRIDE; }

template <int NPROD>
static cudaError_t set_tc_attributes()
{
    // the whole unified L1 as shared memory, so that the two CTAs that tensor memory allows fit on every tree
    cudaError_t e = cudaFuncSetAttribute(k_prune_tc<NPROD>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
        e = allow_smem<k_prune_tc<NPROD>>();
    return e;
}

// CTAs of dynamic shared memory smem that fit an SM: the smaller of what shared memory and
// registers allow (from the kernel's attributes and the device limits) and what tensor memory allows
static int ctas_that_fit(size_t smem)
{
    cudaFuncAttributes fa, fa1;
    int dev = 0, smem_sm = 0, regs_sm = 0, reserved = 0;
    if (cudaFuncGetAttributes(&fa, k_prune_tc<3>) != cudaSuccess || cudaFuncGetAttributes(&fa1, k_prune_tc<1>) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
        return 1;
    const size_t stat = fa.sharedSizeBytes > fa1.sharedSizeBytes ? fa.sharedSizeBytes : fa1.sharedSizeBytes;
    const int regs = fa.numRegs > fa1.numRegs ? fa.numRegs : fa1.numRegs;
    int n = (int)(512 / TCP_TMEM_COLS);
    n = std::min(n, (int)((size_t)smem_sm / (stat + smem + (size_t)reserved)));
    n = std::min(n, regs_sm / (regs * TCP_THREADS));
    return n > 0 ? n : 1;
}

// shapes: 0 = every CTA that fits an SM (two), 1 = one
int prune_tc_ctas_per_sm(int nl, int nint, int shape)
{
    return shape == 1 ? 1 : ctas_that_fit(prune_tc_smem_bytes(nl, nint));
}

size_t prune_tc_stack_floats(int grid, int depth) { return (size_t)grid * prune_tc_levels(depth) * 32 * TCP_THREADS; }

template <int NPROD>
static cudaError_t launch_tc(const PruneArgs &a, float *stack, int *err, cudaStream_t s, int grid)
{
    const size_t smem = prune_tc_smem_bytes(a.nl, a.n_internal);
    cudaError_t e = set_tc_attributes<NPROD>();
    if (e != cudaSuccess) return e;
    k_prune_tc<NPROD><<<grid, TCP_THREADS, smem, s>>>(a, stack, err);
    return cudaGetLastError();
}

cudaError_t launch_prune_tc(int nprod, const PruneArgs &a, float *stack, int *err, cudaStream_t s, int grid)
{
    if (a.nwi <= 0) return cudaSuccess;
    return nprod == 3 ? launch_tc<3>(a, stack, err, s, grid) : launch_tc<1>(a, stack, err, s, grid);
}

}  // namespace pcsf
