// Internal declarations shared by the host runtime and the CUDA kernels.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/phylocsf_engine.h"

namespace pcsf {

constexpr int K = 64;          // codon states (Code.Codon64.dim)
constexpr int K2 = K * K;
constexpr int MAX_LEAVES = 512;

// One internal node of the pruning schedule, in evaluation order.  A child
// slot of -1 means the child is a leaf (its partial is a one-hot gather).
struct SchedNode {
    int16_t node, lc, rc;
    int8_t lslot, rslot, oslot, pad;
};
static_assert(sizeof(SchedNode) == 10, "SchedNode layout");

// A distinct (model, tree scale) pair: one set of P(t) matrices for every branch.
struct PSet {
    int32_t model;
    int32_t pad;
    double rho;
};

// A likelihood evaluation: region, model (0 coding / 1 noncoding), tree scale,
// and the index of its P set within the launch chunk.
struct Request {
    int32_t region;
    int32_t model;
    int32_t pset;
    uint32_t start;    // low 32 bits of the region's first global column (set by the launcher)
    double rho;
};

// A pruning work item: a tile of columns of one request's region.
struct WorkItem {
    int32_t request;   // index into the launch's request array
    int32_t ncols;     // columns in this tile (<= tile width)
    int64_t col0;      // first global column of the tile
};

// Device view of the two models' eigensystems (all arrays [2][...]).
constexpr int WLIST = 4;
struct DevModels {
    const double *U;        // [2][K][K]  eigenvectors of D^1/2 Q D^-1/2 (columns)
    const float *Uf;        // [2][K][K]  FP32 copy
    const double *lam;      // [2][K]
    const double *sq;       // [2][K]     sqrt(pi)
    const double *isq;      // [2][K]     1/sqrt(pi)
    const double *wrow;     // [2][K]     w_m = sum_j U_jm sqrt(pi_j)  (row-sum identity)
    const int16_t *wlist;   // [2][WLIST] the m with w_m != 0, -1 padded; wlist[0] = -2: more than WLIST
    const double *prior;    // [2][K]     root prior
    const double *wlog;     // [2][K]     prior_a * log(prior_a)
    double tol;             // Q.Diag tol (1e-6)
    // FP32 P(t) formation: E(t) = E(t_g) + D^-1/2 U diag(e^{lam t} - e^{lam t_g}) U^T D^1/2
    // around the nearest point t_g of a geometric grid whose E(t_g) were formed
    // in FP64; below the first grid point E(t) = t Q + t^2/2 Q^2.
    const float *gridT;     // [2][G][K][K]  E(t_g)^T in FP32
    const double *grid_t;   // [G]
    const float *grid_eg;   // [2][G][K]     e^{lam_m t_g}
    int grid_n;
    double grid_lr;         // log of the grid ratio
    const float *Qf;        // [2][K][K]  Q (row-major)
    const float *Q2f;       // [2][K][K]  Q^2
    int sm_count;           // the device's, for the split of a P(t) launch
};

// Lets Kernel be launched with any dynamic shared memory that fits beside its static share.  The limit
// belongs to the kernel, not to a launch, and engines on different threads launch one kernel with
// different sizes (trees, branches per CTA): with a launch's own size here, another thread could lower
// the limit before the launch.  Every thread sets the same value.
constexpr int SMEM_OPTIN = 232448;      // sm_103a: shared memory of a block, at most
template <auto Kernel> inline cudaError_t allow_smem()
{
    static std::atomic<int> limit{0};   // the kernel's, once known
    int n = limit.load(std::memory_order_relaxed);
    if (n == 0) {
        cudaFuncAttributes fa;
        const cudaError_t e = cudaFuncGetAttributes(&fa, Kernel);
        if (e != cudaSuccess) return e;
        n = SMEM_OPTIN - (int)fa.sharedSizeBytes;
        limit.store(n, std::memory_order_relaxed);
    }
    return cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, n);
}

// Status keys: ((branch*K + row) << 4) | code, min-reduced so the first error
// in the reference's (branch, row) order wins.  INT32_MAX = no error.
constexpr int32_t STATUS_NONE = 0x7f7f7f7f;   // what cudaMemset(0x7f) leaves

struct LaunchStats {
    float ms = 0.f;
};

// ---- kernels (kernels.cu) -------------------------------------------------
// Jacobi eigensolver: A [nmat][K][K] symmetric -> U [nmat][K][K], lam [nmat][K].
// cluster = jacobi_cluster(nmat, SMs, jacobi_max_cluster())
cudaError_t launch_jacobi(const double *A, double *U, double *lam, int *status, int nmat, int cluster, cudaStream_t s);
// the largest cluster (of 16, 8) of the eigensolver's CTAs that the current device can place: 16 is
// beyond the portable 8, and whether it fits depends on the SMs left in each processing cluster
int jacobi_max_cluster();
// CTAs per matrix: the largest cluster whose CTAs still have an SM each (the processing clusters' odd
// SMs take one cluster of 8 or 16 off what the SM count alone would allow: on 152 SMs up to 8, 18, 38
// and 76 matrices for 16, 8, 4 and 2)
inline int jacobi_cluster(int nmat, int sm_count, int most)
{
    for (int c = most; c > 1; c /= 2)
        if (nmat <= sm_count / c - (c >= 8 ? 1 : 0)) return c;
    return 1;
}

// P(t) formation for P sets [nps]: writes E^T = (P - I)^T per branch into
// Pbuf ([nps][nbr][K][K], element (j,i) = E[i][j]) in FP64 or FP32.
// raw = true skips the row rule (used to form the FP64 grid itself).
// bop (FP32 only, may be null): tensor-core B operands, [set][nbr - bop_nl][hi, lo][64 x 64],
// of the branches b >= bop_nl (the branches above internal nodes when bop_nl = n_leaves)
// dlo (FP32 only, may be null): [set][nbr][K] low parts of the diagonal of E, so that
// E_ii + dlo_i carries the row rule's diagonal to ~2^-48 (see k_prune)
cudaError_t launch_pform(bool fp64, const PSet *ps, int nps, const double *branch, int nbr,
                         DevModels m, void *Pbuf, int32_t *status_key, cudaStream_t s, bool raw = false,
                         float *bop = nullptr, int bop_nl = 0, float *dlo = nullptr);
cudaError_t launch_d2f(const double *in, float *out, size_t n, cudaStream_t s);
cudaError_t launch_d2f_rows(const double *in, float *out, size_t nmat, int nbr, float *bop, int bop_nl, cudaStream_t s,
                            float *dlo = nullptr, bool leaf_rows = false);
// Leaf codes of an uploaded batch: *first_bad = the smallest index of a byte > 64
// (PCSF_MARGINALIZE), left unchanged when every code is valid.
cudaError_t launch_check_codes(const uint8_t *codes, size_t n, unsigned long long *first_bad, cudaStream_t s);

// Pruning over work items [nwi]; partials [nwi][2] (lpr, elpr).
struct PruneArgs {
    const WorkItem *wi;
    int nwi;
    const Request *req;
    const uint8_t *leaves;   // [total_cols][nl]
    const void *Pbuf;        // per chunk-local P set: [nbr][K][K] E^T
    const SchedNode *sched;  // [n_internal]
    int n_internal;
    int nl;
    int nbr;
    int nslots;
    DevModels m;
    double *partials;        // [nwi][2]
    const void *Bop;         // tensor-core kernel: per chunk-local P set, [nbop][hi, lo][64 x 64] B operands
    int nbop;                //   of the branches above internal nodes (node nl + k)
    int dither;              // SIMT FP32 kernel: per-column dithering of the leaf partials (prune_common.cuh)
    const float *dlo;        // SIMT FP32 kernel, may be null: per chunk-local P set [nbr][K] low parts of diag(E)
    int tile;                // SIMT kernel: column tile PRUNE_SMALL_TILE (short launches), 32 or 64 (FP32), 0 = the default rule
    double *colv;            // SIMT kernel, small tiles: [nwi][tile][2] the columns' terms instead of partials
    int depth;               // tensor-core kernels: partials that wait at once (entries of a CTA's stack)
};
// comp: 0 plain FP32 sums, 1 Kahan, 2 blocked Kahan (see prune_common.cuh)
cudaError_t launch_prune(int prec, int comp, const PruneArgs &a, cudaStream_t s, int grid);
constexpr int PRUNE_SMALL_TILE = 8;   // the SIMT kernel's column tile in a short launch
// Whether a launch of this many small tiles is short.  FP32: while all of them are resident at once, four
// per SM; such a launch is as long as one CTA's walk down the tree, which takes a third to a half of the
// time with a column per thread (64 against 8 columns: 58 leaves, 300 columns 212 / 105 us, 4,800 columns
// 214 / 167; 12 leaves 56 / 33 and 57 / 52; 120 leaves, 32 against 8 columns, 302 / 193 and 302 / 322).  FP64 is bound by its two
// lanes per clock and SM at any tile, so that only the balance counts, up to four long tiles (32 columns)
// an SM: small ones unless the last wave of long ones is more than three quarters full.  The third is no
// exception to them: where two CTAs share an SM, it does not spread evenly.  Measured with 32 and 8
// columns, ms at 2,424 / 4,856 / 7,288 / 9,720 / 12,152 / 14,584 / 17,016 / 19,448 columns: 12 leaves 0.41,
// 0.41, 0.79, 0.79, 1.17, 1.56, 1.57, 1.57 and 0.21, 0.50, 0.60, 0.89, 1.09, 1.19, 1.48, 1.68; 58 leaves
// 2.17, 2.16, 4.32, 4.32, 6.48, 6.48, 8.64, 8.63 and 1.09, 2.17, 3.25, 4.33, 5.41, 6.49, 7.57, 8.65.
inline int64_t small_tiles_most(bool fp64, int sm_count) { return (fp64 ? 16 : 4) * (int64_t)sm_count; }
inline bool small_tiles(bool fp64, int64_t tiles, int sm_count)
{
    if (tiles > small_tiles_most(fp64, sm_count)) return false;
    if (!fp64 || tiles == 0) return true;
    const int64_t wave = 4 * (int64_t)sm_count, waves = (tiles + wave - 1) / wave;
    return waves == 3 || 4 * (tiles - (waves - 1) * wave) <= 3 * wave;
}
int prune_tile_cols(int prec);
int simt_tile_cols(int prec, int nslots, int tile = 0);   // the SIMT kernel's column tile (k_prune)
size_t prune_smem_bytes(int prec, int nslots, int nl, int nint, int tile = 0);

// Adjoint gradient over work items (grad_kernels.cu): per work item the lpr /
// elpr partials and d lpr / d t_c for every branch c.
struct GradArgs {
    const WorkItem *wi;
    int nwi;
    const Request *req;
    const uint8_t *leaves;
    const void *Pbuf;
    const SchedNode *sched;
    int n_internal;
    int nl;
    int nbr;
    int nslots;
    DevModels m;
    const void *Qrow;        // [model][K][K] Q row-major in the arithmetic type
    void *scratch;           // gridDim.x * scratch_per_cta bytes
    size_t scratch_per_cta;
    double *partials;        // [nwi][2]
    double *gpart;           // [nwi][nbr + npar]
    // rate-matrix parameter derivatives (OmegaModel kappa, omega): d lpr / d x =
    // sum_c sum_col inter_c^T (dP_c / dx) alpha_c / z, with dP/dx = D^-1/2 U (F o Bdot_x) U^T D^1/2
    int npar;                // 0 or 2
    const void *Hmat;        // [pset][nbr][npar][K][K] (F(t_c) o Bdot_x)^T, arithmetic type
    const void *Umat;        // [model][K][K] U row-major, arithmetic type
    int recompute_leaves;    // leaf children's partials recomputed in the outside pass, not stored
};
cudaError_t launch_grad(int prec, int comp, const GradArgs &a, cudaStream_t s, int grid);
size_t grad_scratch_per_cta(int prec, int nl, int npar, bool recompute_leaves);
size_t grad_smem_bytes(int prec, int nslots, int nl, int nint, int npar);   // the limit on trees
int grad_tile_cols();
int grad_ctas_per_sm(int prec, int nslots, int nl, int nint, int npar);
// H_x = (F(t) o Bdot_x)^T for every (P set, branch, parameter): F_ij = (e^{lam_i t} - e^{lam_j t}) /
// (lam_i - lam_j), t e^{lam_i t} on the diagonal (Frechet derivative of exp in the eigenbasis)
cudaError_t launch_hform(bool fp64, const PSet *ps, int nps, const double *branch, int nbr, const double *lam,
                         const void *Bdot, void *H, cudaStream_t s);
// OmegaModel models keys [nmodels][12] with eigenvectors U and sqrt(pi), 1/sqrt(pi): Q row-major and
// Bdot_x = U^T D^1/2 (dQ/dx) D^-1/2 U, x = kappa, omega, [nmodels][2], in the arithmetic type
cudaError_t launch_omega_deriv(bool fp64, const double *keys, const double *U, const double *sq, const double *isq, int nmodels,
                               void *Q, void *Bdot, cudaStream_t s);
// codon counts of each region's leaves, hist [nreg][64]; offs [nreg + 1] column offsets
cudaError_t launch_codon_hist(const uint8_t *codes, const int64_t *offs, int nreg, int nl, unsigned long long *hist, cudaStream_t s);
cudaError_t launch_reduce_grad(const double *gpart, const int32_t *wi_begin, int nreq, int nbr, double *grad,
                               cudaStream_t s);

// Tensor-core pruning (tc_kernels.cu): nprod 3 = TF32 hi/lo split, 1 = single TF32.
// stack = prune_tc_stack_floats(grid, depth) floats.
cudaError_t launch_prune_tc(int nprod, const PruneArgs &a, float *stack, int *err, cudaStream_t s, int grid);
size_t prune_tc_smem_bytes(int nl, int nint);
size_t prune_tc_stack_floats(int grid, int depth);
bool prune_tc_supported(int nslots, int nl);
constexpr int PCSF_TC_SHAPES = 2;      // 0 every CTA that fits an SM (two), 1 one per SM (identical values)
int prune_tc_ctas_per_sm(int nl, int nint, int shape);
bool prune_tc_shape_ok(int shape);
// Tensor-core pruning with BF16 split products (tc_bf16.cu): x = h + m + l, six
// products on tcgen05 kind::f16, FP32 accumulation; E^T of every branch in Pbuf (FP32).
cudaError_t launch_prune_bf16(const PruneArgs &a, int *err, cudaStream_t s, int grid);
size_t prune_bf16_smem_bytes(int nl, int nint);
bool prune_bf16_supported(int nslots, int nl);
int prune_bf16_ctas_per_sm(int nslots, int nl, int nint);
// tensor-core P(t) formation for the search evaluations (tc_pform.cu): E^T of the
// branches above leaves into Pbuf, B operands of the branches above internal
// nodes into Bop (leaf_rows, here and in launch_d2f_rows: for the branches above leaves
// P^T = E^T + I instead, in the order that k_prune_tc gathers, leaf_pos); Bpf = per model
// the pre-split B = U^T D^1/2 [2][hi, lo][64 x 64]
cudaError_t launch_pform_tc(const PSet *ps, int nps, const double *branch, int nbr, int nl, DevModels m,
                            const float *Bpf, float *Pbuf, float *Bop, int32_t *status_key, int *err, cudaStream_t s,
                            bool leaf_rows = false);
// tensor-core tangent pass (tc_dual.cu): lpr / elpr partials as k_prune_tc plus
// d lpr / d rho partials dpart [nwi][2] (second entry 0); Qop = per model the
// pre-split B operand of Q [2][hi, lo][64 x 64]; branch = the tree's lengths
cudaError_t launch_prune_tc_dual(const PruneArgs &a, const float *Qop, const double *branch, double *dpart, int *err,
                                 cudaStream_t s, int grid);
size_t prune_tc_dual_smem_bytes(int nl, int nint);
bool prune_tc_dual_supported(int nslots, int nl);

// Sum the partials of each request's contiguous work items in fixed order.
// out_index (may be null): request r's sums go to out_*[out_index[r]] instead of out_*[r].
cudaError_t launch_reduce(const double *partials, const int32_t *wi_begin, int nreq, double *out_lpr,
                          double *out_elpr, cudaStream_t s, const int32_t *out_index = nullptr);

// The same from the columns' terms of small tiles (PruneArgs.colv): tc the tile, group the tile
// of a long launch, whose order of summation is kept.
cudaError_t launch_reduce_cols(const double *colv, const WorkItem *wi, const int32_t *wi_begin, int nreq, int tc, int group,
                               double *out_lpr, double *out_elpr, cudaStream_t s);

// Float-float pruning on the tensor cores (ff_kernels.cu): returned values that agree with
// the FP64 path to ~1e-12 relative.  Pbuf holds per P set ff_pset_bytes() of operands, made
// from the FP64 P(t) formation's output by launch_split_ff; tiles of ff_tile_cols() columns,
// one CTA per SM; stack = ff_stack_floats(grid, PruneArgs.depth) floats; partials as
// k_prune; err is set if a bounded wait timed out.
cudaError_t launch_prune_ff(const PruneArgs &a, float *stack, int *err, cudaStream_t s, int grid);
cudaError_t launch_split_ff(const double *in, void *out, int nps, int nbr, int nl, cudaStream_t s);
int ff_tile_cols();
size_t ff_pset_bytes(int nl, int nbr);
size_t ff_stack_floats(int grid, int depth);
size_t prune_ff_smem_bytes(int nl, int nint);

// Outside-pass products (outside_kernels.cu): per request the log-likelihood, optionally the
// expected substitution counts of every branch and the posteriors of selected nodes.  A launch takes
// the work items (tiles of outside_tile_cols() columns) [wi0, wi1) of those that wi holds; the sums
// over a request's tiles go on from one launch to the next, so that they do not depend on where the
// launches end.
struct OutsideArgs {
    const WorkItem *wi;          // work items, contiguous per request
    const int32_t *wi_begin;     // [nreq + 1]
    int wi0, wi1;
    int nreq;
    const Request *req;          // Request.pset indexes Pbuf
    const uint8_t *leaves;       // [total_cols][nl]
    const void *Pbuf;            // E^T sets [nps][nbr][K2] (float or double)
    const SchedNode *sched;
    int n_internal, nl, nbr, nslots;
    DevModels m;
    void *scratch;               // gridDim.x * scratch_per_cta bytes
    size_t scratch_per_cta;
    double *tile_lpr;            // [work items]
    double *lpr;                 // [nreq]
    void *tile_counts;           // [wi1 - wi0][nbr][K][K] (float or double), one launch's
    double *counts;              // [nreq][nbr][K][K]; null: none
    const int32_t *sel;          // [n] output row of each node, -1 if not selected; null: no posteriors
    double *post;                // [n_selected][total_cols][K]
    int64_t total_cols;
};
cudaError_t launch_outside(bool fp64, int comp, const OutsideArgs &a, cudaStream_t s, int grid);
int outside_tile_cols();
int outside_ctas_per_sm(bool fp64, int comp, int nslots, int nl, int nint);
size_t outside_smem_bytes(bool fp64, int nslots, int nl, int nint);
size_t outside_scratch_per_cta(bool fp64, int nl);

// Read-only view of an engine's device state for the allocation-free entry point
// (noalloc.cu; filled by engine.cpp).
struct NoallocCtx {
    int device;
    cudaStream_t stream;
    int prec;              // PCSF_PREC_*
    int comp;              // summation mode of the returned-value kernel (as pcsf_lpr uses it)
    bool pt64;             // P(t) formed in FP64 and rounded to FP32 (PCSF_PT_FP64)
    bool tc_direct;        // pcsf_lpr returns tensor-core values (PCSF_TC_DIRECT)
    bool has_models;
    int nl, nbr, n_internal, nslots;
    const double *branch;
    const SchedNode *sched;
    DevModels m;
    int prune_grid;
    int simt_tile;         // SIMT column tile chosen for the engine (0: the default rule)
    int ff_grid;           // CTAs of the float-float kernel (0: not available)
    int depth;             // its stack: entries per CTA, and the memory
    float *ff_stack;
    int64_t exact_min_units;   // regions with columns x (nl - 2) >= this use the float-float kernel
    int *derr;             // device error flag of timed-out waits
};

}  // namespace pcsf
