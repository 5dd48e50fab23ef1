// Float-float pruning on the tensor cores: returned likelihoods that agree with the
// FP64 path to about 1e-12 relative.
//
// The FP32 kernels round every stored partial and every contraction to 24 bits.
// Over a long region those errors add up partly coherently (columns that share
// sub-patterns repeat them), and the model's P(t) stored in FP32 is itself a fixed
// perturbation that every column sees; together they grow linearly with the
// region's length, past 1e-3 dB at a few thousand codons on trees of ~100 leaves.
// This kernel instead carries every partial as an unevaluated sum of two floats
// (hi + lo, ~48 bits) and contracts it exactly:
//   - E = P - I comes from the FP64 P(t) formation (the FP64 engine's own matrices, row
//     rule of Q.ml:226-247 applied in FP64).  Once per P set (k_split_ff) each row of a
//     branch above an internal node is written as its diagonal in hi / lo floats and its
//     off-diagonal entries as 2^ea sum_l e_l 2^(-8-9l), seven signed 9-bit digits (an error
//     below 2^-63 of the largest of them), and each branch above a leaf as P in hi / lo floats;
//   - a partial alpha, normalised per column to [0.5, 1), becomes sum_k A_k 2^(-8-9k), seven
//     signed 9-bit digits (an error below 2^-60 of the column's largest entry);
//   - sum_{j != a} E[a][j] alpha[j] = 2^(ea-16) sum_g 2^(-9g) G_g with G_g = sum_{k+l=g} sum_j
//     e_l[a][j] A_k[j], kept for g <= 7 (34 of the 49 digit products; the rest are below
//     2^-63).  Digits are FP16 operands of tcgen05.mma kind::f16 (at most 9 bits + sign of
//     FP16's 11); the products of a group share one FP32 accumulator in tensor memory and
//     are integers whose sums stay below 2^24 for g <= 3 (64 x 2^16 x 4 pairs) and, in any
//     case, round by 2^-52 or less beyond, where the digits' signs keep them far below 2^24:
//     so the accumulation is exact, and it does not matter in which order or with which
//     rounding the tensor cores add;
//   - the groups are summed, and alpha and the diagonal's term added (v = alpha + E alpha,
//     PhyloLik.ml:89-92), with error-free transforms; a leaf child's partial is a gathered row of P
//     (PhyloLik.ml:87-88 with a one-hot leaf);
//   - node products alpha = v_l * v_r are float-float products;
//   - each column is rescaled by an exact power of two after every node;
//   - the root dot with the prior, the log and the tile sums are FP64.
// Splitting an operand into digits whose products a low-precision unit adds without
// error is Ozaki's scheme (Ozaki, Ogita, Oishi, Rump 2012).  The error-free steps use
// explicitly rounded add / sub / mul / fma on pairs (f32x2: the same lanes per clock as
// scalar FP32 at half the issue slots), which the compiler never contracts.
//
// Shape: one CTA of 512 threads per SM and 128-column tile; thread t owns column t % 128
// (its TMEM lane) and states 16 (t / 128) .. + 15.  A_k (7 x 16 KB) and the e_l of one
// branch (56 KB, one bulk copy, fetched while the previous contraction is combined) sit in
// shared memory.  B's rows are ordered [digit l][state], so one MMA of A_k against the
// first digits of B adds into consecutive groups: D column 32 g + state for half of the
// states at a time, so the first half is combined while the second half's MMAs run.
// The node evaluated just before its parent is handed over in registers; the other
// internal child (a first child whose sibling is internal) waits on a per-thread stack in
// global memory (L2).
// What bounds it: the chain of a contraction's phases, 14,700 clocks on 120 leaves (13,700 with
// six digits, of which: digits 1,900, staging barrier 1,100, first half's MMAs 2,700 (with the
// sibling leaf's gather), its combination beside the second half's MMAs 2,300, the second half's
// 2,000, the maximum and rescale 500, and per node 3,200 of leaf gathers and stack traffic); a
// third of the issue slots are used.  The MMAs need 4,450 clocks, and a float-float dot product
// on the FP32 units (64 x 12 instructions per state and column instead of about 65) took 75,000.
// Measured per column and evaluation: 120 leaves 238 -> 48 ns, 100 leaves 210 -> 39, 58 leaves 133
// -> 25 (23 in launches that fill the GPU).
// Why seven digits: they are counted from a row's and a column's largest entries.  In a column
// whose two halves of the tree hold codons three substitutions apart, the entries that matter
// lie 2^-20 and more below those.  Against the FP64 engine on the same P(t), the lpr of such a
// column on 58 leaves is off by 1e-14, 3e-14 and 2e-13 at rho = 1, 0.1 and 0.01 (with six digits
// 1e-12, 1e-11 and 1e-10); the FP64 formation of P(t) itself leaves 8e-12, 7e-11 and 7e-10 there.
// The lpr of regions is within 6e-16 relative at rho >= 1 and 5e-14 at rho = 0.01, where two
// independent FP64 evaluations differ by 2e-12.
#include <algorithm>

#include <cuda_fp16.h>

#include "pcsf_internal.h"
#include "prune_common.cuh"
#include "tc_common.cuh"

namespace pcsf {

namespace {

constexpr int FF_THREADS = 512;
constexpr int FF_TC = 128;           // columns per tile
constexpr int FF_DIG = 7;            // 9-bit digits per operand
constexpr int FF_GRP = 8;            // digit groups k + l = 0 .. 7
constexpr int FF_BROWS = 32 * FF_DIG;   // rows of B: [digit][32 states]
constexpr int FF_SPT = 16;           // states per thread
constexpr size_t FF_LEAF_BYTES = 2 * K2 * sizeof(float);            // P of a leaf branch, [s][hi 64 | lo 64]
constexpr uint32_t FF_HALF_BYTES = FF_BROWS * K * 2;                // e_l of 32 states: 224 rows x 64, FP16
constexpr size_t FF_INNER_BYTES = 2 * FF_HALF_BYTES;
constexpr uint32_t FF_ROW_BYTES = 3 * K * 4;                        // per row: scale 2^(ea - 16), E_aa hi, E_aa lo

// dynamic shared memory (bytes)
constexpr uint32_t FS_A = 0;                                        // [digit][128 x 64] FP16
constexpr uint32_t FS_ADIG = 128 * K * 2;
constexpr uint32_t FS_B = FS_A + FF_DIG * FS_ADIG;                  // [half][224 x 64] FP16
constexpr uint32_t FS_SC = FS_B + 2 * FF_HALF_BYTES;                // [2][3][64] row scales and diagonals
constexpr uint32_t FS_CM = FS_SC + 2 * FF_ROW_BYTES;                       // [2][4][128] column maxima
constexpr uint32_t FS_LV = FS_CM + 2 * 4 * FF_TC * 4;               // [nl][128] leaf states (if they fit), schedule, order

// byte offset of (leaf l, site c): words XOR-swizzled per leaf, so that the fill (consecutive
// threads on consecutive leaves) and the reads (on consecutive sites) are free of conflicts
__device__ __forceinline__ int ff_lv(int l, int c) { return l * FF_TC + (c ^ ((l & 31) << 2)); }

size_t ff_smem(int nl, int nint, bool lv)
{
    return FS_LV + (lv ? (size_t)nl * FF_TC : 0) + (size_t)nint * (sizeof(SchedNode) + 2) + 16;
}
// a tile's leaf states are kept in shared memory where the tree leaves them room (up to 362 leaves)
bool ff_lv_fits(int nl, int nint) { return ff_smem(nl, nint, true) + 4096 <= (size_t)SMEM_OPTIN; }

// s + e = a + b exactly (Knuth)
__device__ __forceinline__ void two_sum2(f2 a, f2 b, f2 &s, f2 &e)
{
    s = add2(a, b);
    const f2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
// the same when |a| >= |b| (or a == 0) (Dekker)
__device__ __forceinline__ void fast_two_sum2(f2 a, f2 b, f2 &s, f2 &e)
{
    s = add2(a, b);
    e = sub2(b, sub2(s, a));
}
// s + e = a + G c exactly, for a group's sum G (an integer below 2^24) with weight c and the sum a of the
// groups before, a multiple of 512 c: if |s| < 2^24 c, s is not rounded; beyond, a - s is a multiple of
// s's last place and at most 2^24 c, a float either way, and what G c has left over it one too
__device__ __forceinline__ void add_group(f2 a, f2 G, f2 c, f2 &s, f2 &e)
{
    s = fma2(G, c, a);
    e = fma2(G, c, sub2(a, s));
}
// two FP16 values from a pair of floats that hold small integers (exact)
__device__ __forceinline__ uint32_t half2_of(f2 a)
{
    float x, y;
    upk(a, x, y);
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}

// float-float product of (ah, al) and (bh, bl)
__device__ __forceinline__ void ff_mul2(f2 ah, f2 al, f2 bh, f2 bl, f2 &h, f2 &l)
{
    const f2 p = mul2(ah, bh);
    f2 lo = fma2(ah, bh, neg2(p));
    lo = fma2(ah, bl, lo);
    lo = fma2(al, bh, lo);
    fast_two_sum2(p, lo, h, l);
}

// Seven signed 9-bit digits of a pair x = h + l in [0, 1): x = sum_k d_k 2^(-8-9k).  Rounding to
// an integer by adding 1.5 x 2^23; the residual r is kept negated, so that each digit comes out
// as magic - t without a sign flip.  l joins before digit 2 (error-free: r is 0 or a multiple of h's
// last place, at least twice l, so that r - s is exact; the sum's error e joins
// the residual of digit 3: rounded there by at most 2^-61).
__device__ __forceinline__ void ff_digits(f2 h, f2 l, uint32_t d[FF_DIG])
{
    const f2 M = pk(12582912.0f, 12582912.0f), S = pk(512.0f, 512.0f);
    const f2 x = mul2(h, pk(-256.0f, -256.0f));
    f2 nd = sub2(M, add2(x, M));
    d[0] = half2_of(nd);
    f2 r = add2(x, nd);
    nd = sub2(M, fma2(r, S, M));
    d[1] = half2_of(nd);
    r = fma2(r, S, nd);
    const f2 ml = pk(-131072.0f, -131072.0f), s = fma2(l, ml, r), e = fma2(l, ml, sub2(r, s));      // units 2^-17
    nd = sub2(M, fma2(s, S, M));
    d[2] = half2_of(nd);
    r = fma2(s, S, nd);
    nd = sub2(M, fma2(r, S, M));
    d[3] = half2_of(nd);
    r = fma2(r, S, nd);
    r = fma2(e, pk(262144.0f, 262144.0f), r);
    nd = sub2(M, fma2(r, S, M));
    d[4] = half2_of(nd);
    r = fma2(r, S, nd);
    nd = sub2(M, fma2(r, S, M));
    d[5] = half2_of(nd);
    r = fma2(r, S, nd);
    d[6] = half2_of(sub2(M, fma2(r, S, M)));
}

__device__ __forceinline__ void mma_f16(uint32_t dt, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 :: "r"(dt), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}

// four columns of each of the eight groups (32 columns apart), and the wait, in one asm block
__device__ __forceinline__ void tmem_ld_groups(uint32_t ta, float g[FF_GRP][4])
{
    uint32_t r[FF_GRP * 4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%32];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%33];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%34];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%35];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16,%17,%18,%19}, [%36];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%37];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24,%25,%26,%27}, [%38];\n"
                 "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%28,%29,%30,%31}, [%39];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(ta), "r"(ta + 32), "r"(ta + 64), "r"(ta + 96), "r"(ta + 128), "r"(ta + 160), "r"(ta + 192),
                   "r"(ta + 224)
                 : "memory");
#pragma unroll
    for (int k = 0; k < FF_GRP; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) g[k][j] = __uint_as_float(r[4 * k + j]);
}

// Split of FP64 E^T sets [nps][nbr][K2] into the operands of k_prune_ff, one CTA per matrix.
// Per P set: the leaf branches' P, the inner branches' digits, the inner branches' row scales
// (ff_pset_bytes).  FP64 instructions are the scarce ones (two lanes per clock): two per entry.
__global__ void __launch_bounds__(256) k_split_ff(const double *in, unsigned char *out, int nbr, int nl, size_t pset_bytes)
{
    __shared__ int emax[4][K];
    const int tid = threadIdx.x, a = tid & (K - 1), qd = tid >> 6;      // row a, columns 16 qd ..
    const int b = blockIdx.x % nbr;
    const double *src = in + (size_t)blockIdx.x * K2;
    unsigned char *base = out + (size_t)(blockIdx.x / nbr) * pset_bytes;
    double x[16];
#pragma unroll
    for (int j = 0; j < 16; j++) x[j] = src[(16 * qd + j) * K + a];     // E[a][16 qd + j]
    if (b < nl) {
        float *dst = reinterpret_cast<float *>(base + (size_t)b * FF_LEAF_BYTES);
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int s = 16 * qd + j;
            const double p = x[j] + (a == s ? 1.0 : 0.0);
            const float h = (float)p;
            dst[(size_t)s * 2 * K + a] = h;
            dst[(size_t)s * 2 * K + K + a] = (float)(p - (double)h);
        }
        return;
    }
    float *row = reinterpret_cast<float *>(base + (size_t)nl * FF_LEAF_BYTES + (size_t)(nbr - nl) * FF_INNER_BYTES +
                                           (size_t)(b - nl) * FF_ROW_BYTES);
    // ea: every off-diagonal |E[a][j]| < 2^ea (at least 2^-110, so that the scale stays a normal
    // float); the diagonal, hundreds of times the entries that matter beside it, is kept apart
    int hi = 0;
#pragma unroll
    for (int j = 0; j < 16; j++) {
        if (16 * qd + j == a) {
            const float d = (float)x[j];
            row[K + a] = d;
            row[2 * K + a] = (float)(x[j] - (double)d);
            x[j] = 0.0;
        }
        hi = max(hi, __double2hiint(x[j]) & 0x7fffffff);
    }
    emax[qd][a] = hi;
    __syncthreads();
    hi = max(max(emax[0][a], emax[1][a]), max(emax[2][a], emax[3][a]));
    const int ea = max((hi >> 20) - 1022, -110);
    const double up = __hiloint2double((1023 + 9 * FF_DIG - 1 - ea) << 20, 0);
    const int half = (a >> 3) & 1, n0 = (a >> 4) * 8 + (a & 7);         // state 16 q + 8 half + i -> row 8 q + i
    unsigned char *dst = base + (size_t)nl * FF_LEAF_BYTES + (size_t)(b - nl) * FF_INNER_BYTES + half * FF_HALF_BYTES;
#pragma unroll
    for (int c = 0; c < 2; c++) {                                       // 8 columns: one core-matrix row of 16 bytes
        uint32_t w[FF_DIG][4];
#pragma unroll
        for (int j2 = 0; j2 < 4; j2++) {
            long long v[2];
#pragma unroll
            for (int u = 0; u < 2; u++) v[u] = __double2ll_rn(x[8 * c + 2 * j2 + u] * up);
#pragma unroll
            for (int l = FF_DIG - 1; l >= 0; l--) {
                uint32_t hb = 0;
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int d = l ? (int)((v[u] + 256) & 511) - 256 : (int)v[u];
                    v[u] = (v[u] - d) >> 9;
                    hb |= (uint32_t)__half_as_ushort(__int2half_rn(d)) << (16 * u);
                }
                w[l][j2] = hb;
            }
        }
#pragma unroll
        for (int l = 0; l < FF_DIG; l++) {
            const int n = 32 * l + n0;
            *reinterpret_cast<uint4 *>(dst + (((2 * qd + c) * (FF_BROWS / 8) + (n >> 3)) << 7) + ((n & 7) << 4)) =
                make_uint4(w[l][0], w[l][1], w[l][2], w[l][3]);
        }
    }
    if (qd == 0) row[a] = __int_as_float((127 + ea - 16) << 23);
}

__global__ void __launch_bounds__(FF_THREADS, 1) k_prune_ff(PruneArgs a, size_t pset_bytes, float *stack, int *err, int lv_smem)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint32_t tbase_s;
    __shared__ __align__(8) uint64_t bar_h0, bar_h1, bar_b;
    __shared__ double prd[K], wld[K];
    __shared__ double red_l[4], red_e[4];
    __shared__ int nbseq_s;

    const int tid = threadIdx.x, warp = tid >> 5;
    const int site = tid & (FF_TC - 1);          // tile column = TMEM lane
    const int h = tid >> 7, s0 = FF_SPT * h;      // states s0 .. s0 + 15
    const int nl = a.nl, nin = a.n_internal;
    uint8_t *lvT = sm + FS_LV;
    SchedNode *sched = reinterpret_cast<SchedNode *>(sm + FS_LV + (lv_smem ? nl * FF_TC : 0));
    int16_t *bseq = reinterpret_cast<int16_t *>(sched + nin);        // internal child of each contraction, in order
    const uint32_t bar0 = smem_addr(&bar_h0), bar1 = smem_addr(&bar_h1), barB = smem_addr(&bar_b);
    const uint32_t sA = smem_addr(sm + FS_A), sB = smem_addr(sm + FS_B);
    float *stk = stack + (size_t)blockIdx.x * a.depth * (2 * FF_SPT * FF_THREADS) + tid;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&tbase_s)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar0), "r"(1));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar1), "r"(1));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(barB), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // contraction order: the child evaluated just before its parent (handed over in
        // registers), then the child that waits on the stack
        int k = 0;
        for (int f = 0; f < nin; f++) {
            const SchedNode sn = a.sched[f];
            const int prev = f ? a.sched[f - 1].node : -1;
            const bool li = sn.lslot >= 0, ri = sn.rslot >= 0;
            if (li && ri) {
                bseq[k++] = prev == sn.lc ? sn.lc : sn.rc;
                bseq[k++] = prev == sn.lc ? sn.rc : sn.lc;
            } else if (li || ri) {
                bseq[k++] = li ? sn.lc : sn.rc;
            }
        }
        nbseq_s = k;
    }
    for (int f = tid; f < nin; f += FF_THREADS) sched[f] = a.sched[f];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = tbase_s;
    const int nbseq = nbseq_s;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    ContractionPhase ph_d;              // both D halves complete once per contraction
    uint32_t ph_b = 0;
    int ld_w = blockIdx.x, ld_k = 0, ld_n = 0;   // next B load: work item, index into bseq, loads issued
    int b_inflight = 0;
    int cn = 0;                          // contractions so far (parity: the row-scale buffer)
    bool ok = true;
    const size_t inner0 = (size_t)nl * FF_LEAF_BYTES, scale0 = inner0 + (size_t)(a.nbr - nl) * FF_INNER_BYTES;

    auto issue_next_b = [&]() {          // thread 0: the B buffer is free
        while (ld_w < a.nwi && ld_k >= nbseq) { ld_w += gridDim.x; ld_k = 0; }
        if (ld_w >= a.nwi || nbseq == 0) return;
        const unsigned char *ps = static_cast<const unsigned char *>(a.Pbuf) +
                                  (size_t)a.req[a.wi[ld_w].request].pset * pset_bytes;
        const int c = bseq[ld_k++] - nl;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(barB), "r"((uint32_t)FF_INNER_BYTES + FF_ROW_BYTES) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(sB), "l"(ps + inner0 + (size_t)c * FF_INNER_BYTES), "r"((uint32_t)FF_INNER_BYTES), "r"(barB)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(smem_addr(sm + FS_SC) + (uint32_t)(ld_n & 1) * FF_ROW_BYTES), "l"(ps + scale0 + (size_t)c * FF_ROW_BYTES),
                        "r"(FF_ROW_BYTES), "r"(barB)
                     : "memory");
        ld_n++;
        b_inflight++;
    };
    if (tid == 0) issue_next_b();

    // thread 0, after the staging barrier: the digit products of one contraction.  Operand
    // layouts: K-major core matrices (8 rows x 16 bytes); A_k 128 rows: 2048 B between core
    // matrices along K, B 224 rows: 3584 B; a K step (16 values) is two of them.
    auto issue_mma = [&]() {
        const uint64_t dA = sdesc(sA, 2048, 128), dB = sdesc(sB, FF_BROWS * 16, 128);
        const uint32_t id0 = (1u << 4) | ((128u >> 4) << 24);     // f32 += f16 x f16, M = 128
#pragma unroll 1
        for (int hf = 0; hf < 2; hf++) {
            const uint32_t dt = tbase + 32 * FF_GRP * hf;
            const uint64_t dBh = dB + (FF_HALF_BYTES >> 4) * hf;
            // the first K step starts every group: groups 1-7 by A_1 x e_0..6, group 0 by A_0 x e_0
            mma_f16(dt + 32, dA + (FS_ADIG >> 4), dBh, id0 | ((uint32_t)(FF_BROWS >> 3) << 17), 0);
            mma_f16(dt, dA, dBh, id0 | ((32u >> 3) << 17), 0);
            mma_f16(dt + 32, dA, dBh + (32 * 16 >> 4), id0 | ((uint32_t)((FF_BROWS - 32) >> 3) << 17), 1);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
#pragma unroll
                for (int k = 0; k < FF_DIG; k++) {
                    if (ks == 0 && k < 2) continue;
                    const uint32_t n = 32u * (k == 0 ? FF_DIG : FF_GRP - k);
                    mma_f16(dt + 32 * k, dA + (FS_ADIG >> 4) * k + 256 * ks, dBh + (FF_BROWS * 2) * ks, id0 | ((n >> 3) << 17), 1);
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(hf ? bar1 : bar0) : "memory");
        }
    };
    // this thread's 16 states of a leaf branch's P: v (or v *=) P[.][s], 1 where marginalised
    auto leaf_rows = [&](const unsigned char *P, int s, float *xh, float *xl) {
        const float *row = reinterpret_cast<const float *>(P) + (size_t)(s < K ? s : 0) * 2 * K + s0;
        ldg8(row, xh);
        ldg8(row + 8, xh + 8);
        ldg8(row + K, xl);
        ldg8(row + K + 8, xl + 8);
#pragma unroll
        for (int j = 0; j < FF_SPT; j++) {
            xh[j] = (s < K) ? xh[j] : 1.0f;
            xl[j] = (s < K) ? xl[j] : 0.0f;
        }
    };

    for (int w = blockIdx.x; w < a.nwi && ok; w += gridDim.x) {
        const WorkItem wi = a.wi[w];
        const Request rq = a.req[wi.request];
        const int md = rq.model;
        const unsigned char *Pbase = static_cast<const unsigned char *>(a.Pbuf) + (size_t)rq.pset * pset_bytes;
        const int ncols = wi.ncols;
        const uint8_t *lg = a.leaves + (size_t)wi.col0 * nl;
        __syncthreads();
        if (lv_smem)
            for (int f = tid; f < FF_TC * nl; f += FF_THREADS) {
                const int c = f / nl, l = f - c * nl;
                lvT[ff_lv(l, c)] = (c < ncols) ? lg[f] : (uint8_t)K;
            }
        auto leaf_state = [&](int l) -> int {
            if (lv_smem) return lvT[ff_lv(l, site)];
            return site < ncols ? lg[(size_t)site * nl + l] : K;
        };
        if (tid < K) {
            prd[tid] = a.m.prior[md * K + tid];
            wld[tid] = a.m.wlog[md * K + tid];
        }
        __syncthreads();
        int escale = 0;          // this column's sum of rescale exponents
        int sp = 0;              // stack entries in use
        bool bad = false;        // a timed-out wait not yet agreed on
        f2 ah[FF_SPT / 2], al[FF_SPT / 2];      // the last node's partial

        for (int ni = 0; ni < nin && ok; ni++) {
            const SchedNode sn = sched[ni];
            const int nint = (sn.lslot >= 0) + (sn.rslot >= 0);
            f2 vh[FF_SPT / 2], vl[FF_SPT / 2];
            bool have = false;
            if (nint == 0) {
                float xh[FF_SPT], xl[FF_SPT], yh[FF_SPT], yl[FF_SPT];
                leaf_rows(Pbase + (size_t)sn.lc * FF_LEAF_BYTES, leaf_state(sn.lc), xh, xl);
                leaf_rows(Pbase + (size_t)sn.rc * FF_LEAF_BYTES, leaf_state(sn.rc), yh, yl);
#pragma unroll
                for (int i = 0; i < FF_SPT / 2; i++)
                    ff_mul2(pk(xh[2 * i], xh[2 * i + 1]), pk(xl[2 * i], xl[2 * i + 1]), pk(yh[2 * i], yh[2 * i + 1]),
                            pk(yl[2 * i], yl[2 * i + 1]), vh[i], vl[i]);
            }
            for (int c = 0; c < nint; c++) {
                if (c == 1) {                   // the waiting child, back from the stack
                    sp--;
                    const float *st = stk + (size_t)sp * (2 * FF_SPT * FF_THREADS);
#pragma unroll
                    for (int i = 0; i < FF_SPT / 2; i++) {
                        ah[i] = pk(st[(2 * i) * FF_THREADS], st[(2 * i + 1) * FF_THREADS]);
                        al[i] = pk(st[(FF_SPT + 2 * i) * FF_THREADS], st[(FF_SPT + 2 * i + 1) * FF_THREADS]);
                    }
                }
                // ---- digits of alpha: the A operand (free: the last contraction's MMAs completed)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    uint32_t d[4][FF_DIG];
#pragma unroll
                    for (int i = 0; i < 4; i++) ff_digits(ah[4 * q + i], al[4 * q + i], d[i]);
                    const uint32_t o = (uint32_t)((((s0 >> 3) + q) * 16 + (site >> 3)) << 7) + ((site & 7) << 4);
#pragma unroll
                    for (int k = 0; k < FF_DIG; k++)
                        *reinterpret_cast<uint4 *>(sm + FS_A + FS_ADIG * k + o) = make_uint4(d[0][k], d[1][k], d[2][k], d[3][k]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (tid == 0) {
                    if (mbar_wait(barB, ph_b)) b_inflight--;
                    else bad = true;
                }
                tc_fence_before();
                if (__syncthreads_or(bad)) { ok = false; break; }
                tc_fence_after();
                ph_b ^= 1u;
                if (tid == 0) issue_mma();
                if (nint == 1) {                // the leaf beside it, gathered while the MMAs run
                    const int lc = (sn.lslot < 0) ? sn.lc : sn.rc;
                    float xh[FF_SPT], xl[FF_SPT];
                    leaf_rows(Pbase + (size_t)lc * FF_LEAF_BYTES, leaf_state(lc), xh, xl);
#pragma unroll
                    for (int i = 0; i < FF_SPT / 2; i++) {
                        vh[i] = pk(xh[2 * i], xh[2 * i + 1]);
                        vl[i] = pk(xl[2 * i], xl[2 * i + 1]);
                    }
                    have = true;
                }
                // ---- v (or v *=) alpha + E alpha, half of the states at a time
                const float *sc = reinterpret_cast<const float *>(sm + FS_SC) + (cn & 1) * 3 * K + s0;
#pragma unroll
                for (int hf = 0; hf < 2; hf++) {
                    if (!mbar_wait(hf ? bar1 : bar0, ph_d.wait())) bad = true;
                    tc_fence_after();
                    if (hf == 1 && tid == 0 && !bad) issue_next_b();     // every MMA of B has completed
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        float g[FF_GRP][4];
                        tmem_ld_groups(tbase + lane_off + 32 * FF_GRP * hf + 8 * h + 4 * q, g);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const int x = 4 * hf + 2 * q + i;            // pair of states s0 + 2 x, s0 + 2 x + 1
                            f2 G[FF_GRP];
#pragma unroll
                            for (int k = 0; k < FF_GRP; k++) G[k] = pk(g[k][2 * i], g[k][2 * i + 1]);
                            const f2 c9 = pk(0x1p-9f, 0x1p-9f);
                            f2 s1, e1, s2, e2, s3, e3, s4, e4;
                            add_group(G[0], G[1], c9, s1, e1);
                            add_group(s1, G[2], pk(0x1p-18f, 0x1p-18f), s2, e2);
                            add_group(s2, G[3], pk(0x1p-27f, 0x1p-27f), s3, e3);
                            add_group(s3, G[4], pk(0x1p-36f, 0x1p-36f), s4, e4);
                            const f2 L = fma2(fma2(G[7], c9, G[6]), c9, G[5]);
                            const f2 lo = add2(add2(e1, e2), add2(e3, fma2(L, pk(0x1p-45f, 0x1p-45f), e4)));
                            const f2 scale = *reinterpret_cast<const f2 *>(sc + 2 * x);
                            // + (alpha + E_aa alpha), the largest terms: three float-float numbers
                            const f2 dh = *reinterpret_cast<const f2 *>(sc + K + 2 * x);
                            const f2 dl = *reinterpret_cast<const f2 *>(sc + 2 * K + 2 * x);
                            const f2 p = mul2(dh, ah[x]);
                            f2 pl = fma2(dh, ah[x], neg2(p));
                            pl = fma2(dh, al[x], pl);
                            pl = fma2(dl, ah[x], pl);
                            f2 t, e, u, f, uh, ul;
                            fast_two_sum2(ah[x], p, t, e);      // |E_aa| < 1
                            two_sum2(t, mul2(s4, scale), u, f);
                            fast_two_sum2(u, add2(add2(al[x], pl), add2(e, fma2(lo, scale, f))), uh, ul);
                            if (have) ff_mul2(vh[x], vl[x], uh, ul, vh[x], vl[x]);
                            else { vh[x] = uh; vl[x] = ul; }
                        }
                    }
                }
                ph_d.next();
                cn++;
                have = true;
            }
            if (!ok) break;
            // ---- column maximum over the four threads of a column, rescale by an exact power of two
            float mx = 0.0f;
#pragma unroll
            for (int i = 0; i < FF_SPT / 2; i++) {
                float x, y;
                upk(vh[i], x, y);
                mx = fmaxf(mx, fmaxf(x, y));
            }
            float *cm = reinterpret_cast<float *>(sm + FS_CM) + (ni & 1) * 4 * FF_TC;
            cm[h * FF_TC + site] = mx;
            // the four warps that share these columns: a named barrier (1-4) of those 128 threads
            asm volatile("bar.sync %0, 128;" :: "r"(1 + (warp & 3)) : "memory");
            mx = fmaxf(fmaxf(cm[site], cm[FF_TC + site]), fmaxf(cm[2 * FF_TC + site], cm[3 * FF_TC + site]));
            const int e = (mx > 0.0f) ? exp_of(mx) : 0;
            escale += e;
            const int ehalf = (-e) >> 1;                     // 2^-e as two factors, as scale2
            const float f1 = __int_as_float((ehalf + 127) << 23), f2s = __int_as_float((-e - ehalf + 127) << 23);
            const f2 p1 = pk(f1, f1), p2 = pk(f2s, f2s);
#pragma unroll
            for (int i = 0; i < FF_SPT / 2; i++) {
                ah[i] = mul2(mul2(vh[i], p1), p2);
                al[i] = mul2(mul2(vl[i], p1), p2);
            }
            // not a child of the next node: it waits on the stack
            if (ni + 1 < nin && sched[ni + 1].lc != sn.node && sched[ni + 1].rc != sn.node) {
                float *st = stk + (size_t)sp * (2 * FF_SPT * FF_THREADS);
#pragma unroll
                for (int i = 0; i < FF_SPT / 2; i++) {
                    float x, y;
                    upk(ah[i], x, y);
                    st[(2 * i) * FF_THREADS] = x;
                    st[(2 * i + 1) * FF_THREADS] = y;
                    upk(al[i], x, y);
                    st[(FF_SPT + 2 * i) * FF_THREADS] = x;
                    st[(FF_SPT + 2 * i + 1) * FF_THREADS] = y;
                }
                sp++;
            }
        }
        if (!ok) break;
        if (__syncthreads_or(bad)) { ok = false; break; }
        // ---- root: z = alpha_root . prior ; elpr term = (alpha_root . prior*log prior) / z, in
        // FP64 (the A operand is idle: partial sums [z, wz][4][128])
        double *zp = reinterpret_cast<double *>(sm + FS_A);
        {
            double z = 0.0, wz = 0.0;
#pragma unroll
            for (int i = 0; i < FF_SPT / 2; i++) {
                float xh[2], xl[2];
                upk(ah[i], xh[0], xh[1]);
                upk(al[i], xl[0], xl[1]);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const double x = (double)xh[u] + (double)xl[u];
                    z += x * prd[s0 + 2 * i + u];
                    wz += x * wld[s0 + 2 * i + u];
                }
            }
            zp[h * FF_TC + site] = z;
            zp[(4 + h) * FF_TC + site] = wz;
        }
        __syncthreads();
        if (h == 0) {
            double tl = 0.0, te = 0.0;
            if (site < ncols) {
                const double z = (zp[site] + zp[FF_TC + site]) + (zp[2 * FF_TC + site] + zp[3 * FF_TC + site]);
                const double wz = (zp[4 * FF_TC + site] + zp[5 * FF_TC + site]) + (zp[6 * FF_TC + site] + zp[7 * FF_TC + site]);
                if (z > 0.0) {
                    tl = log(z) + (double)escale * 0.69314718055994530942;
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
            if ((tid & 31) == 0) {
                red_l[warp] = tl;
                red_e[warp] = te;
            }
        }
        __syncthreads();
        if (tid == 0) {
            a.partials[2 * (size_t)w] = ((red_l[0] + red_l[1]) + red_l[2]) + red_l[3];
            a.partials[2 * (size_t)w + 1] = ((red_e[0] + red_e[1]) + red_e[2]) + red_e[3];
        }
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    // quiesce: a bulk copy may be outstanding (loads run one ahead) and, after a timed-out
    // wait, MMAs; both waits are bounded
    if (tid == 0 && b_inflight > 0 && !mbar_wait(barB, ph_b)) atomicExch(err, 1);
    if (!ok) {
        mbar_wait(bar0, ph_d.last());
        mbar_wait(bar1, ph_d.last());
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(512));
}

}  // namespace

int ff_tile_cols() { return FF_TC; }

size_t ff_pset_bytes(int nl, int nbr)
{
    return (size_t)nl * FF_LEAF_BYTES + (size_t)(nbr - nl) * (FF_INNER_BYTES + FF_ROW_BYTES);
}

size_t ff_stack_floats(int grid, int depth) { return (size_t)grid * std::max(depth, 1) * 2 * FF_SPT * FF_THREADS; }

cudaError_t launch_split_ff(const double *in, void *out, int nps, int nbr, int nl, cudaStream_t s)
{
    if (nps <= 0 || nbr <= 0) return cudaSuccess;
    k_split_ff<<<(unsigned)nps * (unsigned)nbr, 256, 0, s>>>(in, static_cast<unsigned char *>(out), nbr, nl,
                                                             ff_pset_bytes(nl, nbr));
    return cudaGetLastError();
}

size_t prune_ff_smem_bytes(int nl, int nint) { return ff_smem(nl, nint, ff_lv_fits(nl, nint)); }

cudaError_t launch_prune_ff(const PruneArgs &a, float *stack, int *err, cudaStream_t s, int grid)
{
    if (a.nwi <= 0) return cudaSuccess;
    const bool lv = ff_lv_fits(a.nl, a.n_internal);
    const size_t smem = ff_smem(a.nl, a.n_internal, lv);
    cudaError_t e = allow_smem<k_prune_ff>();
    if (e != cudaSuccess) return e;
    k_prune_ff<<<grid, FF_THREADS, smem, s>>>(a, ff_pset_bytes(a.nl, a.nbr), stack, err, lv);
    return cudaGetLastError();
}

}  // namespace pcsf
