// SIMT kernels of the likelihood engine: FP64 eigensolver, P(t) formation,
// Felsenstein pruning (FP64 and FP32) and the per-request reduction.
//
// Reference behaviour restated here (paths relative to mlin/PhyloCSF):
//   eigendecomposition  lib/CamlPaml/Q.ml:124-141 (GSL nonsymmv + complex LU in the
//                       reference; a parallel cyclic Jacobi on D^1/2 Q D^-1/2 here)
//   P(t) + row rule     lib/CamlPaml/Q.ml:211-249
//   inside pass         lib/CamlPaml/PhyloLik.ml:73-93
//   root posterior      lib/CamlPaml/PhyloLik.ml:127-138, src/PhyloCSFModel.ml:67-82
#include <cfloat>
#include <cmath>
#include <cstdio>

#include <cooperative_groups.h>

#include "jacobi_rotation.cuh"
#include "pcsf_internal.h"
#include "prune_common.cuh"

namespace pcsf {

// ---------------------------------------------------------------------------
// Eigensolver: parallel cyclic Jacobi, C CTAs (one cluster) per symmetric 64x64 matrix.
// Each sweep visits all 2016 pairs as 63 rounds of 32 disjoint rotations (round-robin
// "circle" ordering), which are applied simultaneously.
//
// What bounds it: a round is 24,576 FP64 instructions (A <- J^T A J as 1024 blocks of 2x2,
// V <- V J), and an SM issues two FP64 lanes per clock: ~12,300 clocks a round on one SM, 500
// to 600 rounds.  The matrices of a call are few (two models, or one per region of an
// OmegaModel round), so the rows of A and V are spread over a cluster: a block of pair k's
// rows and pair k' 's columns is read from and written to the owners' shared memory, A is
// double-buffered so that a round needs one cluster barrier, and V, whose rows are local, is
// updated between arriving at that barrier and waiting for it.  Every element goes through
// the same operations in the same order for every C: the results do not depend on it.
// Measured, OmegaModel scores of six 12-leaf alignments (130 rounds of up to 8 matrices): 514 ms
// with one CTA per matrix, 243 ms with clusters of 16, 207 ms with small pruning tiles, 181 ms with
// half blocks per thread, their loads ahead of the rotations, and jac_rotation's short chain.  A
// round is ~4,300 clocks now: about 1,500 of rotations and 500 of updates, the rest distributed
// shared-memory latency and the barrier.

constexpr int JAC_THREADS = 256;
constexpr int JAC_LD = K + 1;

__device__ inline void jac_pair(int r, int i, int &p, int &q)
{
    int a, b;
    if (i == 0) { a = K - 1; b = r; }
    else { a = (r + i) % (K - 1); b = (r - i + (K - 1)) % (K - 1); }
    p = a < b ? a : b;
    q = a < b ? b : a;
}

template <int C>
__global__ void __launch_bounds__(JAC_THREADS) k_jacobi(const double *A_in, double *U_out, double *lam_out,
                                                         int *status)
{
    constexpr int ROWS = K / C;                        // rows of A and V per CTA
    constexpr int HALVES = (32 / C) * 64;              // half blocks of a CTA: two per pair of pairs
    constexpr bool HALF = HALVES <= JAC_THREADS;       // one per thread (C >= 8)
    extern __shared__ __align__(16) unsigned char jsm[];
    double *A = reinterpret_cast<double *>(jsm);      // [2][ROWS][JAC_LD]
    double *V = A + 2 * ROWS * JAC_LD;                 // [ROWS][JAC_LD]
    double *red = V + ROWS * JAC_LD;                   // [JAC_THREADS]
    double *csb = red + JAC_THREADS;                   // [2][32]
    double *snb = csb + 64;                            // [2][32]
    int *ppb = reinterpret_cast<int *>(snb + 64);      // [2][32]
    int *qqb = ppb + 64;                               // [2][32]
    const int tid = threadIdx.x;
    const int rank = blockIdx.x % C, row0 = rank * ROWS;
    const double *Ain = A_in + (size_t)(blockIdx.x / C) * K2;

    auto cluster_arrive = [&]() {
        if constexpr (C > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    };
    auto cluster_wait = [&]() {
        if constexpr (C > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        else __syncthreads();
    };
    // a x - b y and a x + b y, the second product rounded (fixed here so that every form of the
    // update rounds alike)
    auto diff = [](double a, double x, double b, double y) { return __fma_rn(a, x, -__dmul_rn(b, y)); };
    auto sum = [](double a, double x, double b, double y) { return __fma_rn(a, x, __dmul_rn(b, y)); };
    // element (row, col) of buffer buf, wherever it lives in the cluster
    auto at = [&](int buf, int row, int col) -> double * {
        double *p = A + ((size_t)buf * ROWS + row % ROWS) * JAC_LD + col;
        if constexpr (C > 1) p = cooperative_groups::this_cluster().map_shared_rank(p, row / ROWS);
        return p;
    };

    for (int f = tid; f < ROWS * K; f += JAC_THREADS) {
        const int i = f / K, j = f % K;
        A[i * JAC_LD + j] = Ain[(row0 + i) * K + j];
        V[i * JAC_LD + j] = (row0 + i == j) ? 1.0 : 0.0;
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    // ||A||_F^2 (fixed-order tree reduction)
    double part = 0.0;
    for (int f = tid; f < K2; f += JAC_THREADS) {
        double x = Ain[f];
        part += x * x;
    }
    red[tid] = part;
    __syncthreads();
    for (int w = JAC_THREADS / 2; w > 0; w >>= 1) {
        if (tid < w) red[tid] += red[tid + w];
        __syncthreads();
    }
    const double norm2 = red[0];
    __syncthreads();

    int converged = 0, cur = 0;
    for (int sweep = 0; sweep < 60; sweep++) {
        part = 0.0;
        for (int f = tid; f < K2; f += JAC_THREADS) {
            int i = f / K, j = f % K;
            if (i < j) { double x = *at(cur, i, j); part += x * x; }
        }
        red[tid] = part;
        __syncthreads();
        for (int w = JAC_THREADS / 2; w > 0; w >>= 1) {
            if (tid < w) red[tid] += red[tid + w];
            __syncthreads();
        }
        double off = red[0];
        __syncthreads();
        if (off <= 1e-32 * norm2) { converged = 1; break; }     // the same in every CTA of the cluster
        for (int r = 0; r < K - 1; r++) {
            double *cs = csb + 32 * (cur & 1), *sn = snb + 32 * (cur & 1);
            int *pp = ppb + 32 * (cur & 1), *qq = qqb + 32 * (cur & 1);
            // HALF: a thread's half block, one of the two columns of pair kc in the rows of pair k, is
            // on its way while the rotations are formed
            double x[4];
            if (HALF && tid < HALVES) {
                int p, q, pc, qc;
                jac_pair(r, rank * (32 / C) + (tid >> 6), p, q);
                jac_pair(r, tid & 31, pc, qc);
                x[0] = *at(cur, p, pc);
                x[1] = *at(cur, p, qc);
                x[2] = *at(cur, q, pc);
                x[3] = *at(cur, q, qc);
            }
            if (tid < 32) {                                     // every CTA forms all 32 rotations
                int p, q;
                jac_pair(r, tid, p, q);
                const double apq = *at(cur, p, q), aqq = *at(cur, q, q), app = *at(cur, p, p);
                double c = 1.0, s = 0.0;
                if (apq != 0.0) jac_rotation(app, aqq, apq, c, s);
                cs[tid] = c; sn[tid] = s; pp[tid] = p; qq[tid] = q;
            }
            __syncthreads();
            // 2x2 blocks: columns A <- A J, then rows A <- J^T A (16 FP64 instructions a block); the
            // pivots become exact zeros
            auto column = [&](int k, int kc, bool second) {
                const int p = pp[k], q = qq[k];
                const double cc = cs[kc], sc = sn[kc], cr = cs[k], sr = sn[k];
                if (!second) {
                    const int pc = pp[kc];
                    const double bp = diff(cc, x[0], sc, x[1]), bq = diff(cc, x[2], sc, x[3]);
                    *at(cur ^ 1, p, pc) = diff(cr, bp, sr, bq);
                    *at(cur ^ 1, q, pc) = k == kc ? 0.0 : sum(sr, bp, cr, bq);
                } else {
                    const int qc = qq[kc];
                    const double bp = sum(sc, x[0], cc, x[1]), bq = sum(sc, x[2], cc, x[3]);
                    *at(cur ^ 1, p, qc) = k == kc ? 0.0 : diff(cr, bp, sr, bq);
                    *at(cur ^ 1, q, qc) = sum(sr, bp, cr, bq);
                }
            };
            if (HALF) {
                if (tid < HALVES) column(rank * (32 / C) + (tid >> 6), tid & 31, (tid & 32) != 0);
            } else {
                for (int f = tid; f < HALVES / 2; f += JAC_THREADS) {
                    const int k = rank * (32 / C) + (f >> 5), kc = f & 31;
                    const int p = pp[k], q = qq[k], pc = pp[kc], qc = qq[kc];
                    x[0] = *at(cur, p, pc);
                    x[1] = *at(cur, p, qc);
                    x[2] = *at(cur, q, pc);
                    x[3] = *at(cur, q, qc);
                    column(k, kc, false);
                    column(k, kc, true);
                }
            }
            cluster_arrive();
            for (int f = tid; f < ROWS * 32; f += JAC_THREADS) {       // V <- V J
                const int row = f >> 5, k = f & 31;
                const int p = pp[k], q = qq[k];
                const double c = cs[k], s = sn[k];
                const double va = V[row * JAC_LD + p], vb = V[row * JAC_LD + q];
                V[row * JAC_LD + p] = diff(c, va, s, vb);
                V[row * JAC_LD + q] = sum(s, va, c, vb);
            }
            cluster_wait();
            cur ^= 1;
        }
    }
    __syncthreads();
    double *Uo = U_out + (size_t)(blockIdx.x / C) * K2;
    for (int f = tid; f < ROWS * K; f += JAC_THREADS) Uo[row0 * K + f] = V[(f / K) * JAC_LD + f % K];
    if (tid < ROWS) lam_out[(size_t)(blockIdx.x / C) * K + row0 + tid] = A[(cur * ROWS + tid) * JAC_LD + row0 + tid];
    if (rank == 0 && tid == 0) status[blockIdx.x / C] = converged ? 0 : 1;
    if (C > 1) {                       // no CTA leaves while another may still read its rows
        cluster_arrive();
        cluster_wait();
    }
}

template <int C>
static cudaError_t config_jacobi_c(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &attr, int nmat, cudaStream_t s)
{
    const size_t smem = sizeof(double) * (3 * (K / C) * JAC_LD + JAC_THREADS + 128) + sizeof(int) * 128;
    cudaError_t err = allow_smem<k_jacobi<C>>();
    if (err == cudaSuccess && C > 8)
        err = cudaFuncSetAttribute(k_jacobi<C>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return err;
    cfg.gridDim = dim3(nmat * C);
    cfg.blockDim = dim3(JAC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    return cudaSuccess;
}

template <int C>
static cudaError_t launch_jacobi_c(const double *A, double *U, double *lam, int *status, int nmat, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    const cudaError_t err = config_jacobi_c<C>(cfg, attr, nmat, s);
    return err == cudaSuccess ? cudaLaunchKernelEx(&cfg, k_jacobi<C>, A, U, lam, status) : err;
}

int jacobi_max_cluster()
{
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    int n = 0;
    if (config_jacobi_c<16>(cfg, attr, 1, nullptr) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, k_jacobi<16>, &cfg) == cudaSuccess && n > 0)
        return 16;
    cudaGetLastError();
    return 8;
}

cudaError_t launch_jacobi(const double *A, double *U, double *lam, int *status, int nmat, int cluster, cudaStream_t s)
{
    if (nmat <= 0) return cudaSuccess;
    switch (cluster) {
    case 16: return launch_jacobi_c<16>(A, U, lam, status, nmat, s);
    case 8: return launch_jacobi_c<8>(A, U, lam, status, nmat, s);
    case 4: return launch_jacobi_c<4>(A, U, lam, status, nmat, s);
    case 2: return launch_jacobi_c<2>(A, U, lam, status, nmat, s);
    default: return launch_jacobi_c<1>(A, U, lam, status, nmat, s);
    }
}

// ---------------------------------------------------------------------------
// P(t) formation.  For branch b of request r at t = rho_r * b_b:
//   E = P(t) - I = D^-1/2 U diag(expm1(lam t)) U^T D^1/2
// (expm1 in FP64; the 64^3 product in the storage precision T), then the row
// rule of Q.ml:226-247 on P = I + E:
//   - the raw row sum must be within tol of 1 (evaluated in FP64 through the
//     eigensystem identity sum_j E_ij = isq_i sum_m U_im expm1(lam_m t) w_m);
//   - off-diagonal negatives within tol are set to 0, below -tol are an error;
//   - the diagonal becomes 1 - sum of the off-diagonal entries, and must lie in
//     (0,1].
// Output is E^T: Pbuf[(r*nbr + b)*K2 + j*K + i] = E[i][j].

constexpr int PF_THREADS = 256;
constexpr int PF_BRANCHES = 2;   // most branches per CTA (the eigenvectors are staged once)
constexpr int PF_SPREAD = 2 * 4;         // FP32 matrices of a launch, per SM, up to which each gets its own CTA

// shared memory (dynamic): U^T, with FP64 U^T times the coefficients, per branch E^T and the coefficients
template <typename T> __host__ __device__ constexpr size_t pform_smem(int per_cta)
{
    return sizeof(T) * ((size_t)(sizeof(T) == 8 ? 2 : 1) * K2 + 2 * K + (size_t)per_cta * (K2 + K)) +
           sizeof(double) * (size_t)per_cta * K;
}

// The branches of a CTA go through each phase together: coefficients (a thread per branch and
// eigenvalue), products (the whole CTA, branch after branch), the row rule (a thread per branch and
// row: its compensated sum is a chain of 64 dependent steps, which one branch at a time left on two
// of the eight warps) and the stores.  U^T is stored with the 16-byte chunks of row m permuted by
// XOR with m mod 16, so that neither the transposing stores nor the loads of a product step
// conflict by more than 4.  What bounds the FP32 form is the load/store pipe (64 % of its
// wavefronts at four branches per CTA) and FP32 issue: E^T stays in the layout of the grid and of
// the output from the asynchronous copy of E(t_g) to the store, and lanes run along its rows.
// Measured, 301 P sets of 58 leaves: 0.95 ms with E row-major and one branch at a time, 0.82 with
// this, 0.75 with two branches per CTA (four CTAs per SM) instead of four.
template <typename T>
__global__ void __launch_bounds__(PF_THREADS) k_pform(const PSet *ps, const double *branch, int nbr,
                                                       DevModels m, T *Pbuf, int32_t *status_key, int raw,
                                                       float *Bop, int bop_nl, float *dlo, int per_cta)
{
    constexpr bool fp32 = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char psm[];
    T *UT = reinterpret_cast<T *>(psm);     // [K][K]   UT[m][j] = U[j][m] (chunks permuted)
    T *UeT = UT + K2;                         // [K][K]   FP64: UeT[m][i] = U[i][m] * coef_m
    T *sqT = UT + (fp32 ? 1 : 2) * K2;        // [K]
    T *isqT = sqT + K;                        // [K]
    T *cfT = isqT + K;                        // [per_cta][K] product coefficients
    double *ex = reinterpret_cast<double *>(cfT + per_cta * K);   // [per_cta][K] expm1(lam t): row-sum identity
    T *Eall = reinterpret_cast<T *>(ex + per_cta * K);            // [per_cta][K][K] E^T: element (j, i) = E[i][j]
    __shared__ int mode_s[PF_BRANCHES], grid_s[PF_BRANCHES];
    const int tid = threadIdx.x;
    const int r = blockIdx.y;
    const PSet rq = ps[r];
    const int md = rq.model;
    const double *U = m.U + (size_t)md * K2;
    const float *Uf = m.Uf + (size_t)md * K2;
    const double *lam = m.lam + md * K;
    const double *isq = m.isq + md * K;
    const double *wrow = m.wrow + md * K;
    const int b0 = blockIdx.x * per_cta, nb = min(per_cta, nbr - b0);
    auto chunk = [](int c, int mm) { return 4 * (c ^ (mm & 15)); };   // first entry of chunk c (4 entries) of row mm

    for (int f = tid; f < K2; f += PF_THREADS) {
        int j = f / K, mm = f % K;   // U[j][mm]
        UT[mm * K + chunk(j >> 2, mm) + (j & 3)] = fp32 ? (T)Uf[f] : (T)U[f];
    }
    if (tid < K) {
        sqT[tid] = (T)m.sq[md * K + tid];
        isqT[tid] = (T)isq[tid];
    }
    const int ty = tid % 16, tx = tid / 16;     // rows 4 ty .. (lanes), columns 4 tx .. of E
    // per branch of this CTA, in parallel (one thread each; FP64 is a narrow pipe here):
    // 0: direct eigen formula (FP64);  1: t == 0;  2: Taylor below the grid;  3: grid correction
    if (tid < nb) {
        int mode = 0, g = 0;
        if (fp32 && m.grid_n > 0) {
            const double t = rq.rho * branch[b0 + tid];
            if (t == 0.0) mode = 1;
            else if (t < m.grid_t[0]) mode = 2;
            else {
                mode = 3;
                g = grid_point(m, t);
            }
        }
        mode_s[tid] = mode;
        grid_s[tid] = g;
    }
    __syncthreads();
    // E(t_g), as it is stored, into the place of E^T
    for (int bi = 0; bi < nb; bi++)
        if (mode_s[bi] == 3) {
            const float *base = m.gridT + ((size_t)md * m.grid_n + grid_s[bi]) * K2;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Eall + (size_t)bi * K2);
            for (int f = tid; f < K2 / 4; f += PF_THREADS)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(dst + 16 * f), "l"(base + 4 * f) : "memory");
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int f = tid; f < nb * K; f += PF_THREADS) {
        const int bi = f / K, mm = f % K, mode = mode_s[bi];
        const double t = rq.rho * branch[b0 + bi];
        // ex feeds the row-sum check, which needs it only where w_m != 0
        // (the stationary direction); the FP32 modes therefore spend one
        // FP64 expm1 per branch instead of 64 (FP64 is a narrow pipe here).
        if (mode == 0) {
            ex[f] = expm1(lam[mm] * t);
            cfT[f] = (T)ex[f];
        } else {
            ex[f] = (wrow[mm] != 0.0) ? (double)expm1f((float)(lam[mm] * t)) : 0.0;   // row-sum check only
            if (mode == 3) {
                // e^{lam t_g} (tabulated) * expm1(lam (t - t_g)) in FP32: the
                // coefficient is rounded to FP32 for the GEMM in any case
                const double h = t - m.grid_t[grid_s[bi]];
                const float eg = m.grid_eg[((size_t)md * m.grid_n + grid_s[bi]) * K + mm];
                cfT[f] = (T)(eg * expm1f((float)(lam[mm] * h)));
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int bi = 0; bi < nb; bi++) {
        T *Es = Eall + (size_t)bi * K2;
        const int mode = mode_s[bi];
        const double t = rq.rho * branch[b0 + bi];
        if (mode == 0 || mode == 3) {
            const T *cf = cfT + bi * K;
            if (!fp32) {
                if (bi) __syncthreads();
                for (int f = tid; f < K2; f += PF_THREADS) UeT[f] = UT[f] * cf[f / K];
                __syncthreads();
            }
            T acc[4][4];
            if constexpr (fp32) {
                f2 s2[4][2];
#pragma unroll
                for (int i = 0; i < 4; i++) s2[i][0] = s2[i][1] = 0ull;
#pragma unroll 4
                for (int mm = 0; mm < K; mm++) {
                    float a[4], bb[4];
                    const float c = cf[mm];
                    Vec4<float>::load(UT + mm * K + chunk(ty, mm), a);
                    Vec4<float>::load(UT + mm * K + chunk(tx, mm), bb);
                    const f2 b01 = pk(bb[0], bb[1]), b23 = pk(bb[2], bb[3]);
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float x = __fmul_rn(a[i], c);
                        const f2 xx = pk(x, x);
                        s2[i][0] = fma2(xx, b01, s2[i][0]);
                        s2[i][1] = fma2(xx, b23, s2[i][1]);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    upk(s2[i][0], acc[i][0], acc[i][1]);
                    upk(s2[i][1], acc[i][2], acc[i][3]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) acc[i][j] = (T)0;
                for (int mm = 0; mm < K; mm++) {
                    T a[4], bb[4];
                    Vec4<T>::load(UeT + mm * K + chunk(ty, mm), a);
                    Vec4<T>::load(UT + mm * K + chunk(tx, mm), bb);
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[i][j] += a[i] * bb[j];
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int jj = 4 * tx + j;
                T *e = Es + jj * K + 4 * ty, g[4], v[4];
                if (mode == 3) Vec4<T>::load(e, g);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    v[i] = acc[i][j] * sqT[jj] * isqT[4 * ty + i];
                    if (mode == 3) v[i] += g[i];
                }
                ColStore<T, 4>::store(e, v);
            }
        } else {
            const float *Qf = m.Qf + (size_t)md * K2, *Q2f = m.Q2f + (size_t)md * K2;
            const T tt = (T)t, h = (T)(0.5 * t * t);
            for (int f = tid; f < K2; f += PF_THREADS) {
                int i = f / K, j = f % K;
                Es[j * K + i] = (mode == 1) ? (T)0 : tt * (T)Qf[f] + h * (T)Q2f[f];
            }
        }
    }
    __syncthreads();
    if (tid < nb * K && !raw) {
        const int bi = tid / K, i = tid % K, b = b0 + bi;
        T *row = Eall + (size_t)bi * K2 + i;      // entry j at row[j * K]
        // raw row sum - 1, in FP64 through the eigensystem
        const double rs = rowsum_minus_one(m, md, i, ex + bi * K);
        // the diagonal is the compensated sum of the stored (rounded)
        // off-diagonal entries, so every stored row of P = I + E sums to 1
        // to within one rounding of the diagonal; a plain FP32 sum here
        // biases lpr by ~1e-4 nats per 3000 codons at rho = 1.  Branch-free in
        // j: i differs per lane, and a branch on j == i would split the warp.
        bool neg = false;
        T diag = (T)0, dc = (T)0;
        const T ntol = (T)(-m.tol), dtol = (T)(-1.0 - m.tol);
        for (int j0 = 0; j0 < K; j0 += 8) {
            T x8[8];           // loaded ahead of the stores below
#pragma unroll
            for (int k = 0; k < 8; k++) x8[k] = row[(j0 + k) * K];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int j = j0 + k;
                const bool dj = (j == i);
                const T x0 = x8[k];
                neg |= dj ? (x0 < dtol) : (x0 < ntol);   // diagonal: x + 1 < -tol
                const T x = (x0 < (T)0) ? (T)0 : x0;      // an off-diagonal negative within tol becomes 0
                if (!dj && x != x0) row[j * K] = x;
                if (fp32) {           // Kahan: diag -= x
                    const T y = -x - dc;
                    const T tt = diag + y;
                    const T c = (tt - diag) - y;
                    diag = dj ? diag : tt;
                    dc = dj ? dc : c;
                } else {
                    diag = dj ? diag : diag - x;
                }
            }
        }
        if (neg) status_min(status_key + r, b, i, PCSF_ENEGP);
        else if (fabs(rs) > m.tol) status_min(status_key + r, b, i, PCSF_EROWSUM);
        else if (!(diag > (T)-1)) status_min(status_key + r, b, i, PCSF_EDIAG);
        // the sum is diag - dc to second order: its low part for the pruning kernel
        if (fp32 && dlo) dlo[((size_t)r * nbr + b) * K + i] = (float)(-dc);
        row[i * K] = diag;
    }
    __syncthreads();
    for (int bi = 0; bi < nb; bi++) {
        const int b = b0 + bi;
        const T *Es = Eall + (size_t)bi * K2;
        T *out = Pbuf + ((size_t)r * nbr + b) * K2;
        for (int f = tid; f < (int)(K2 * sizeof(T) / 16); f += PF_THREADS)
            reinterpret_cast<uint4 *>(out)[f] = reinterpret_cast<const uint4 *>(Es)[f];
        if (fp32 && Bop && b >= bop_nl) {      // branch above an internal node: tensor-core operand too
            float *dst = Bop + ((size_t)r * (nbr - bop_nl) + (b - bop_nl)) * 2 * K2;
            for (int f = tid; f < K2 / 4; f += PF_THREADS) {
                const int a = f & (K - 1), q = f >> 6;
                const T *col = Es + 4 * q * K + a;
                bop_store(dst, a, q, make_float4((float)col[0], (float)col[K], (float)col[2 * K], (float)col[3 * K]));
            }
        }
    }
}

cudaError_t launch_pform(bool fp64, const PSet *req, int nreq, const double *branch, int nbr, DevModels m,
                         void *Pbuf, int32_t *status_key, cudaStream_t s, bool raw, float *bop, int bop_nl, float *dlo)
{
    if (nreq <= 0) return cudaSuccess;
    // Two branches per CTA share the staged eigenvectors.  One per CTA where that staging is
    // nothing beside the product (FP64 runs at 1/64 of the FP32 rate: ~70 us per branch) and
    // for short FP32 launches, which more would leave on a part of the SMs.  Measured: FP64,
    // 24 P sets of 29 leaves 0.95 -> 0.69 ms, six of 12 leaves 0.36 -> 0.13 ms; FP32, two P
    // sets of 12 leaves 39 -> 17 us.
    const int per_cta = (fp64 || (int64_t)nreq * nbr <= (int64_t)PF_SPREAD * m.sm_count) ? 1 : PF_BRANCHES;
    dim3 grid((nbr + per_cta - 1) / per_cta, nreq);
    if (fp64) {
        const size_t smem = pform_smem<double>(per_cta);
        cudaError_t e = allow_smem<k_pform<double>>();
        if (e != cudaSuccess) return e;
        k_pform<double><<<grid, PF_THREADS, smem, s>>>(req, branch, nbr, m, (double *)Pbuf, status_key, raw ? 1 : 0,
                                                       nullptr, 0, nullptr, per_cta);
    } else {
        const size_t smem = pform_smem<float>(per_cta);
        cudaError_t e = allow_smem<k_pform<float>>();
        if (e != cudaSuccess) return e;
        k_pform<float><<<grid, PF_THREADS, smem, s>>>(req, branch, nbr, m, (float *)Pbuf, status_key, raw ? 1 : 0,
                                                      bop, bop_nl, raw ? nullptr : dlo, per_cta);
    }
    return cudaGetLastError();
}

__global__ void k_d2f(const double *in, float *out, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

cudaError_t launch_d2f(const double *in, float *out, size_t n, cudaStream_t s)
{
    k_d2f<<<264, 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

// FP64 -> FP32 for E^T matrices that already obey the row rule: off-diagonal
// entries are rounded and each diagonal is re-formed as the FP64 sum of its
// row's rounded entries (storage E^T: element (i, j) of E at [j*K + i]).
// Matrices are [set][nbr]; with bop, the branches b >= bop_nl also get their
// tensor-core B operand (see bop_store).
__global__ void __launch_bounds__(256) k_d2f_rows(const double *in, float *out, size_t nmat, int nbr, float *bop,
                                                  int bop_nl, float *dlo, int leaf_rows)
{
    const size_t mat = blockIdx.x * (size_t)4 + threadIdx.x / K;
    const int i = threadIdx.x % K;
    if (mat >= nmat) return;
    const double *src = in + mat * K2;
    float *dst = out + mat * K2;
    const int b = (int)(mat % (size_t)nbr);
    const bool lr = leaf_rows && b < bop_nl;
    const int pos = lr ? leaf_pos(i) : i;
    double d = 0.0;
    for (int j = 0; j < K; j++) {
        if (j == i) continue;
        const float x = (float)src[j * K + i];
        dst[j * K + pos] = x;
        d -= (double)x;
    }
    dst[i * K + pos] = lr ? (float)d + 1.0f : (float)d;
    if (dlo) dlo[mat * K + i] = (float)(d - (double)(float)d);   // low part of the diagonal
    if (bop && b >= bop_nl) {
        float *bd = bop + ((mat / nbr) * (size_t)(nbr - bop_nl) + (b - bop_nl)) * 2 * K2;
        for (int q = 0; q < K / 4; q++)
            bop_store(bd, i, q, make_float4(dst[(4 * q) * K + i], dst[(4 * q + 1) * K + i], dst[(4 * q + 2) * K + i],
                                            dst[(4 * q + 3) * K + i]));
    }
}

// any byte of w above 64: (b & 0x7F) + 63 reaches bit 7 exactly when b & 0x7F > 64
// (no carry between bytes: at most 190), and b's own bit 7 covers b >= 128
__device__ __forceinline__ bool bytes_above_64(uint32_t w)
{
    return ((((w & 0x7F7F7F7Fu) + 0x3F3F3F3Fu) | w) & 0x80808080u) != 0u;
}

__global__ void k_check_codes(const uint8_t *codes, size_t n, unsigned long long *first_bad)
{
    const size_t t0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    const size_t nv = n / 16;
    for (size_t v = t0; v < nv; v += stride) {
        const uint4 x = reinterpret_cast<const uint4 *>(codes)[v];
        if (bytes_above_64(x.x) || bytes_above_64(x.y) || bytes_above_64(x.z) || bytes_above_64(x.w))
            for (int j = 0; j < 16; j++)
                if (codes[16 * v + j] > 64) {
                    atomicMin(first_bad, (unsigned long long)(16 * v + j));
                    break;
                }
    }
    for (size_t i = 16 * nv + t0; i < n; i += stride)
        if (codes[i] > 64) atomicMin(first_bad, (unsigned long long)i);
}

cudaError_t launch_check_codes(const uint8_t *codes, size_t n, unsigned long long *first_bad, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    size_t blocks = (n / 16 + 255) / 256;
    if (blocks < 1) blocks = 1;
    if (blocks > 4096) blocks = 4096;
    k_check_codes<<<(unsigned)blocks, 256, 0, s>>>(codes, n, first_bad);
    return cudaGetLastError();
}

cudaError_t launch_d2f_rows(const double *in, float *out, size_t nmat, int nbr, float *bop, int bop_nl, cudaStream_t s,
                            float *dlo, bool leaf_rows)
{
    if (nmat == 0) return cudaSuccess;
    k_d2f_rows<<<(unsigned)((nmat + 3) / 4), 256, 0, s>>>(in, out, nmat, nbr, bop, bop_nl, dlo, leaf_rows ? 1 : 0);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Pruning (inside pass).  One CTA (256 threads) owns a tile of TC columns of
// one request's region and walks the internal nodes in the register-minimal
// (Sethi-Ullman) schedule computed on the host; partials live in shared
// memory slots [K][TC].  Thread (ty,tx) owns states 4ty..4ty+3 and columns
// tx*CPT..tx*CPT+CPT-1.
//
// For a child c of node i:   v_c[a] = alpha_c[a] + sum_j E_c[a][j] alpha_c[j]
// (internal child; E = P - I keeps the large diagonal exact; the sum is formed
// first, optionally with compensated summation, and alpha_c[a] added last), or the gather
// v_c[a] = P_c[a][s] for a leaf in state s (1 for a marginalised leaf: P rows
// sum to 1 after the row rule).  Then alpha_i = v_l * v_r, and each column is
// rescaled by an exact power of two so its maximum lies in [0.5,1); the
// exponents are summed per column and added back as e*ln2 in FP64 at the root.

//
// What bounds it: FP32 issue in the contractions (half of the paired FMA rate over a launch) and,
// between them, the phases that the other CTA of the SM covers only in part: the copies of the next
// node's operands (1,400 clocks of a node's 10,000), a leaf's factors (1,300), the rescale (1,000).
// The diagonals' low parts come into L1 with the operands, the leaf states with eight loads in
// flight, and the rescale multiplies once where it can: 58 leaves, 141,741 columns 2.67 -> 2.59 ms,
// 120 leaves, 95,724 columns 4.30 -> 4.17 ms.
constexpr int PR_THREADS = 256;

// threads of a tile: 16 groups of 4 states; 4 or 2 columns per thread, or 1 in half a block (8 columns)
template <int TC> struct PruneThreads { static constexpr int N = TC >= 16 ? PR_THREADS : 16 * TC; };

template <typename T, int TC>
struct PruneSmem {
    static size_t bytes(int nslots, int nl, int nint)
    {
        size_t b = sizeof(T) * (2 * K2 + (size_t)nslots * K * TC);
        b += sizeof(typename AtomMax<T>::U) * 2 * TC;
        b += sizeof(int) * TC;
        b += sizeof(SchedNode) * nint;
        b = (b + 15) & ~size_t(15);
        b += (size_t)nl * TC;
        return (b + 15) & ~size_t(15);
    }
};

template <typename T, int TC, int KAHAN>
__global__ void __launch_bounds__(PruneThreads<TC>::N) k_prune(PruneArgs a)
{
    constexpr int THREADS = PruneThreads<TC>::N, TXN = THREADS / 16, CPT = TC / TXN;
    constexpr bool SMALL = TC == PRUNE_SMALL_TILE;      // a short launch
    typedef typename AtomMax<T>::U MU;
    extern __shared__ __align__(16) unsigned char ssm[];
    T *Et = reinterpret_cast<T *>(ssm);                 // [2][K][K]
    T *slots = Et + 2 * K2;                              // [nslots][K][TC]
    MU *colmax = reinterpret_cast<MU *>(slots + (size_t)a.nslots * K * TC);   // [2][TC]
    int *cscale = reinterpret_cast<int *>(colmax + 2 * TC);                   // [TC]
    SchedNode *sched = reinterpret_cast<SchedNode *>(cscale + TC);            // [n_internal]
    size_t off = (reinterpret_cast<unsigned char *>(sched + a.n_internal) - ssm + 15) & ~size_t(15);
    uint8_t *lvT = ssm + off;                                                  // [nl][TC]

    const int tid = threadIdx.x;
    const int ty = tid / TXN, tx = tid % TXN;
    const int a0 = 4 * ty, c0 = CPT * tx;
    const int nl = a.nl;
    __shared__ double red_l[THREADS / 32], red_e[THREADS / 32];
    __shared__ double ltab[256];           // log(1 + k/256), the dither factors' logs
    __shared__ double dsum[TC];            // per column: sum over leaves of log c
    const bool dith = a.dither && sizeof(T) == 4;

    for (int f = tid; f < a.n_internal; f += THREADS) sched[f] = a.sched[f];
    if (dith)
        for (int f = tid; f < 256; f += THREADS) ltab[f] = log1p((double)f / 256.0);

    for (int w = blockIdx.x; w < a.nwi; w += gridDim.x) {
        const WorkItem wi = a.wi[w];
        const Request rq = a.req[wi.request];
        const int md = rq.model;
        const T *Pbase = reinterpret_cast<const T *>(a.Pbuf) + (size_t)rq.pset * a.nbr * K2;
        // low parts of diag(E) of this P set (FP32 only)
        const float *dlo = (sizeof(T) == 4 && a.dlo) ? a.dlo + (size_t)rq.pset * a.nbr * K : nullptr;
        const int ncols = wi.ncols;
        const uint8_t *lg = a.leaves + (size_t)wi.col0 * nl;
        __syncthreads();   // previous work item finished with shared memory
        // leaf states, eight loads in flight a thread
        for (int f0 = tid; f0 < TC * nl; f0 += 8 * THREADS) {
            uint8_t x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int f = f0 + i * THREADS;
                x[i] = f < ncols * nl ? __ldg(lg + f) : (uint8_t)K;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int f = f0 + i * THREADS, c = f / nl;
                if (f < TC * nl) lvT[(f - c * nl) * TC + c] = x[i];
            }
        }
        for (int f = tid; f < 2 * TC; f += THREADS) colmax[f] = 0;
        for (int f = tid; f < TC; f += THREADS) cscale[f] = 0;
        // dither keys are the column's position within its region, so that results
        // do not depend on where a region sits in the batch
        const int64_t dcol0 = dith ? (int64_t)(uint32_t)((uint32_t)wi.col0 - rq.start) : -1;
        __syncthreads();       // leaf states (and ltab) ready
        // a node's operands are copied one node ahead (issued once the previous node's contraction
        // has released the buffers)
        // and the diagonals' low parts, two lines a child, come into L1 with them
        auto stage = [&](const SchedNode &nx) {
            stage_children<T, TC, CPT, THREADS>(Et, Pbase, nx, lvT, tid);
            if (dlo && tid < 4)
                asm volatile("prefetch.global.L1 [%0];" :: "l"(dlo + (size_t)(tid < 2 ? nx.lc : nx.rc) * K + 32 * (tid & 1)));
        };
        stage(sched[0]);
        if (dith) {
            for (int c = tid; c < TC; c += THREADS) {
                double sd = 0.0;
                for (int l = 0; l < nl; l++) sd += ltab[dither_k(dcol0 + c, l)];
                dsum[c] = sd;
            }
        }

        for (int ni = 0; ni < a.n_internal; ni++) {
            const SchedNode sn = sched[ni];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            T vl[4][CPT], vr[4][CPT];
            child_partial<T, TC, KAHAN, CPT, 7>(Et, slots, sn.lslot, sn.lc, lvT, a0, c0, vl, dcol0, true,
                                        dlo ? dlo + (size_t)sn.lc * K : nullptr);
            child_partial<T, TC, KAHAN, CPT, 7>(Et + K2, slots, sn.rslot, sn.rc, lvT, a0, c0, vr, dcol0, true,
                                        dlo ? dlo + (size_t)sn.rc * K : nullptr);
            __syncthreads();
            if (ni + 1 < a.n_internal) {
                stage(sched[ni + 1]);       // buffers free again
            } else if (SMALL && tid < K) {  // the root's: prior and prior log prior, two doubles a copy
                const double *src = (tid < K / 2 ? a.m.prior : a.m.wlog) + md * K + 2 * (tid % (K / 2));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                             :: "r"((uint32_t)__cvta_generic_to_shared(Et) + 16 * tid), "l"(src) : "memory");
            }
            MU *cm = colmax + (ni & 1) * TC;
            MU *cm_next = colmax + ((ni + 1) & 1) * TC;
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
            T mx[CPT], sc[CPT];
            ColLoad<T, CPT>::load(reinterpret_cast<const T *>(cm) + c0, mx);
            // sc = 2^-e as one factor where every maximum of the warp allows it, else the first of scale2's
            // two factors goes into vl (one column a thread: the test costs what it saves)
            bool one = false;
            if constexpr (sizeof(T) == 4 && CPT > 1) {
                one = true;
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    const int b = __float_as_int(mx[cc]) >> 23;
                    one &= b > 0 && b < 253;
                }
                one = __all_sync(0xffffffffu, one);
                if (one) {
#pragma unroll
                    for (int cc = 0; cc < CPT; cc++) {
                        const int b = __float_as_int(mx[cc]) >> 23;
                        if (ty == 0) cscale[c0 + cc] += b - 126;
                        sc[cc] = __int_as_float((253 - b) << 23);
                    }
                }
            }
            if (!one) {
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) {
                    const int e = (mx[cc] > (T)0) ? exp_of(mx[cc]) : 0, e1 = -e >> 1;
                    if (ty == 0) cscale[c0 + cc] += e;
                    const T first = pow2<T>(e1);
                    sc[cc] = pow2<T>(-e - e1);
#pragma unroll
                    for (int i = 0; i < 4; i++) vl[i][cc] *= first;
                }
            }
            // one vector store per state row (CPT consecutive columns): scalar stores
            // here were 4-way bank-conflicted
#pragma unroll
            for (int i = 0; i < 4; i++) {
                T y[CPT];
#pragma unroll
                for (int cc = 0; cc < CPT; cc++) y[cc] = vl[i][cc] * sc[cc];
                ColStore<T, CPT>::store(out + (a0 + i) * TC + c0, y);
            }
        }
        if (SMALL) asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // root: z = alpha_root . prior ; elpr term = (alpha_root . prior*log prior) / z
        // (in order: a search's parabolic steps magnify the last bit of a value.  A short launch is one
        // CTA's chain, so it has the prior in shared memory and eight steps' loads in flight.)
        double tl = 0.0, te = 0.0;
        if (tid < TC && tid < ncols) {
            const T *ar = slots + (size_t)sched[a.n_internal - 1].oslot * K * TC;
            const double *pr = SMALL ? reinterpret_cast<const double *>(Et) : a.m.prior + md * K;
            const double *wl = SMALL ? pr + K : a.m.wlog + md * K;
            double z = 0.0, wz = 0.0;
#pragma unroll (SMALL ? 8 : 4)
            for (int s = 0; s < K; s++) {
                double x = (double)ar[s * TC + tid];
                z += x * pr[s];
                wz += x * wl[s];
            }
            if (z > 0.0) {
                tl = log(z) + (double)cscale[tid] * 0.69314718055994530942 - (dith ? dsum[tid] : 0.0);
                te = wz / z;
            } else {
                tl = -INFINITY;
                te = 0.0;
            }
        }
        if (a.colv) {      // small tiles: the columns' terms, summed by k_reduce_cols
            if (tid < TC) reinterpret_cast<double2 *>(a.colv)[(size_t)w * TC + tid] = make_double2(tl, te);
            continue;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            tl += __shfl_down_sync(0xffffffffu, tl, o);
            te += __shfl_down_sync(0xffffffffu, te, o);
        }
        if ((tid & 31) == 0) { red_l[tid >> 5] = tl; red_e[tid >> 5] = te; }
        __syncthreads();
        if (tid == 0) {
            double sl = 0.0, se = 0.0;
            for (int k = 0; k < (TC + 31) / 32; k++) { sl += red_l[k]; se += red_e[k]; }
            a.partials[2 * (size_t)w] = sl;
            a.partials[2 * (size_t)w + 1] = se;
        }
    }
}

int prune_tile_cols(int prec)
{
    if (prec == PCSF_PREC_TF32X3 || prec == PCSF_PREC_TF32 || prec == PCSF_PREC_BF16X3) return 128;
    return prec == PCSF_PREC_FP64 ? 32 : 64;
}

// Column tile of the SIMT pruning kernel in a long launch.  FP32 uses 64 columns, except for
// trees of five or more partial slots (the 120-leaf tree): there 64 columns take ~124 KB of
// shared memory, one CTA per SM, and 32 columns let two CTAs share an SM.
// tile (32 or 64) overrides this rule for the FP32 kernel (the engine's autotuner sets it).
int simt_tile_cols(int prec, int nslots, int tile)
{
    if (prec == PCSF_PREC_FP64) return 32;
    if (tile == 32 || tile == 64) return tile;
    return nslots >= 5 ? 32 : 64;
}

template <typename T>
static size_t prune_smem_t(int tc, int nslots, int nl, int nint)
{
    if (tc == PRUNE_SMALL_TILE) return PruneSmem<T, PRUNE_SMALL_TILE>::bytes(nslots, nl, nint);
    if (tc == 32) return PruneSmem<T, 32>::bytes(nslots, nl, nint);
    return PruneSmem<T, 64>::bytes(nslots, nl, nint);
}

size_t prune_smem_bytes(int prec, int nslots, int nl, int nint, int tile)
{
    const int tc = tile == PRUNE_SMALL_TILE ? tile : simt_tile_cols(prec, nslots, tile);
    return prec == PCSF_PREC_FP64 ? prune_smem_t<double>(tc, nslots, nl, nint) : prune_smem_t<float>(tc, nslots, nl, nint);
}

template <typename T, int TC, int KAHAN>
static cudaError_t launch_prune_t(const PruneArgs &a, cudaStream_t s, int grid)
{
    size_t smem = PruneSmem<T, TC>::bytes(a.nslots, a.nl, a.n_internal);
    cudaError_t e = allow_smem<k_prune<T, TC, KAHAN>>();
    if (e != cudaSuccess) return e;
    k_prune<T, TC, KAHAN><<<grid, PruneThreads<TC>::N, smem, s>>>(a);
    return cudaGetLastError();
}

template <int TC>
static cudaError_t launch_prune_f(int comp, const PruneArgs &a, cudaStream_t s, int grid)
{
    if (comp == 1) return launch_prune_t<float, TC, 1>(a, s, grid);
    if (comp == 2) return launch_prune_t<float, TC, 2>(a, s, grid);
    return launch_prune_t<float, TC, 0>(a, s, grid);
}

cudaError_t launch_prune(int prec, int comp, const PruneArgs &a, cudaStream_t s, int grid)
{
    if (a.nwi <= 0) return cudaSuccess;
    if (prec == PCSF_PREC_FP64) {
        if (a.tile == PRUNE_SMALL_TILE) return launch_prune_t<double, PRUNE_SMALL_TILE, 0>(a, s, grid);
        return launch_prune_t<double, 32, 0>(a, s, grid);
    }
    if (a.tile == PRUNE_SMALL_TILE) return launch_prune_f<PRUNE_SMALL_TILE>(comp, a, s, grid);
    if (simt_tile_cols(prec, a.nslots, a.tile) == 32) return launch_prune_f<32>(comp, a, s, grid);
    return launch_prune_f<64>(comp, a, s, grid);
}

// ---------------------------------------------------------------------------
// Per-request sums of the work-item partials, in work-item order (deterministic).

__global__ void k_reduce(const double *partials, const int32_t *wi_begin, int nreq, double *out_lpr, double *out_elpr,
                         const int32_t *out_index)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nreq) return;
    double sl = 0.0, se = 0.0;
    for (int w = wi_begin[r]; w < wi_begin[r + 1]; w++) {
        sl += partials[2 * (size_t)w];
        se += partials[2 * (size_t)w + 1];
    }
    const int o = out_index ? out_index[r] : r;
    out_lpr[o] = sl;
    out_elpr[o] = se;
}

// The same sums from the columns' terms of a launch of small tiles (tc columns, ragged last tile
// per request): per group of `group` columns (the tile of a long launch) a tree over each 32, the
// groups in order -- bit for bit what k_prune and k_reduce form with tiles of that size.  One CTA
// per request: its warps form the trees of up to RC_CHUNKS times 32 columns side by side, two
// threads add them up.  What bounds it: the latency of the loads and of the FP64 additions; a warp
// per request, one tree after the other, took 14 us for a call of 600 columns, 8 us now (a launch
// and its copy included), and 0.25 ms of the 18 rounds of 48 ORFs, 0.19 now.
constexpr int RC_THREADS = 256, RC_PER = 4, RC_CHUNKS = RC_PER * RC_THREADS / 32;
__global__ void __launch_bounds__(RC_THREADS) k_reduce_cols(const double2 *colv, const WorkItem *wi, const int32_t *wi_begin,
                                                            int tc, int group, double *out_lpr, double *out_elpr)
{
    __shared__ double sums[2][RC_CHUNKS];
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w0 = wi_begin[r], w1 = wi_begin[r + 1];
    const int64_t ncols = w1 > w0 ? (int64_t)(w1 - 1 - w0) * tc + wi[w1 - 1].ncols : 0;
    const double2 *src = colv + (size_t)w0 * tc;
    double tot = 0.0;          // threads 0 (lpr) and 32 (elpr)
    for (int64_t c0 = 0; c0 < ncols; c0 += 32 * RC_CHUNKS) {
        double2 t[RC_PER];
#pragma unroll
        for (int i = 0; i < RC_PER; i++) {
            const int64_t c = c0 + 32 * (warp + i * (RC_THREADS / 32)) + lane;
            t[i] = c < ncols ? src[c] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int i = 0; i < RC_PER; i++) {
            const int k = warp + i * (RC_THREADS / 32);
            if (c0 + 32 * k >= ncols) break;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                t[i].x += __shfl_down_sync(0xffffffffu, t[i].x, o);
                t[i].y += __shfl_down_sync(0xffffffffu, t[i].y, o);
            }
            if (lane == 0) {
                sums[0][k] = t[i].x;
                sums[1][k] = t[i].y;
            }
        }
        __syncthreads();
        if (lane == 0 && warp < 2) {
            const int n = (int)min((int64_t)RC_CHUNKS, (ncols - c0 + 31) / 32);
            for (int k = 0; k < n; k += group / 32) {
                double g = 0.0;
                for (int j = k; j < min(n, k + group / 32); j++) g += sums[warp][j];
                tot += g;
            }
        }
        __syncthreads();
    }
    if (lane == 0 && warp < 2) (warp ? out_elpr : out_lpr)[r] = tot;
}

cudaError_t launch_reduce_cols(const double *colv, const WorkItem *wi, const int32_t *wi_begin, int nreq, int tc, int group,
                               double *out_lpr, double *out_elpr, cudaStream_t s)
{
    if (nreq <= 0) return cudaSuccess;
    k_reduce_cols<<<nreq, RC_THREADS, 0, s>>>(reinterpret_cast<const double2 *>(colv), wi, wi_begin, tc, group, out_lpr, out_elpr);
    return cudaGetLastError();
}

cudaError_t launch_reduce(const double *partials, const int32_t *wi_begin, int nreq, double *out_lpr,
                          double *out_elpr, cudaStream_t s, const int32_t *out_index)
{
    if (nreq <= 0) return cudaSuccess;
    k_reduce<<<(nreq + 127) / 128, 128, 0, s>>>(partials, wi_begin, nreq, out_lpr, out_elpr, out_index);
    return cudaGetLastError();
}

}  // namespace pcsf
