// QR-preconditioned one-sided Jacobi SVD (sm_100a): the fast path for tall
// and for ill-conditioned matrices.
//
//   1. A = Q R by shifted CholeskyQR3 (Fukaya, Kannan, Nakatsukasa, Yamamoto,
//      Yanagisawa, SIAM J. Sci. Comput. 2020): one Cholesky QR pass on
//      A^T A + s I, s = 11 (m n + n (n + 1)) u ||A||_F^2, then two plain passes
//      (CholeskyQR2).  Stable for kappa(A) up to about 1/u; Q orthogonal to
//      working precision.
//   2. One-sided Jacobi on X = R^T (n x n) with the plain sweep (same
//      arithmetic, same round-robin order).  For ill-conditioned A the columns
//      of R^T are graded and the sweep count drops (Drmac and Veselic, SIAM J.
//      Matrix Anal. Appl. 29, 2008); for tall A every round also moves m/n
//      times fewer bytes.
//   3. X V_x = U_x Sigma  =>  A = Q R = Q V_x Sigma U_x^T, so
//      V_A = U_x (normalised columns of the rotated X), U_A = Q V_x, Sigma_A =
//      Sigma_x (unsorted, in X's column order).
// Gram products and triangular updates run on this library's FP64 tensor-core
// GEMM (dgemm.cu); the Cholesky diagonal blocks, the triangular row solves,
// the shift and the layout kernels are written here.  If a Cholesky pivot is
// not positive the solve falls back to the plain path on A.
#include <cuda_runtime.h>

#include <atomic>

#include <algorithm>
#include <memory>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "blockpair.hpp"
#include "common.cuh"
#include "dgemm.hpp"
#include "internal.hpp"
#include "jsvd.h"
#include "layout.cuh"
#include "mixed.hpp"
#include "plain.hpp"
#include "ptx.cuh"

namespace jsvd {
namespace {

constexpr int kNb = 64;  // Cholesky / triangular block size

#define JSVD_GEMM_TRY(EXPR)                       \
    do {                                          \
        const int gemm_rc_ = (EXPR);              \
        if (gemm_rc_ != JSVD_OK) return gemm_rc_; \
    } while (0)

// row-major (rows x cols) -> column-major (ld = rows), one launch (the n x n
// factor; the m x n input goes through launch_rowmajor_to_colmajor)
__global__ void __launch_bounds__(kTile *kTileRows)
    pc_to_colmajor(const double *__restrict__ src, int rows, int cols, double *__restrict__ dst)
{
    __shared__ double tile[kTile][kTile + 1];
    const int c0 = blockIdx.x * kTile, r0 = blockIdx.y * kTile;
    for (int k = threadIdx.y; k < kTile; k += kTileRows) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        if (r < rows && c < cols) tile[k][threadIdx.x] = src[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < kTile; k += kTileRows) {
        const int c = c0 + k, r = r0 + threadIdx.x;
        if (r < rows && c < cols) dst[(size_t)c * rows + r] = tile[threadIdx.x][k];
    }
}

// G_ii += s with s = 11 (m n + n (n + 1)) u trace(G)   (one CTA)
__global__ void __launch_bounds__(256) pc_shift_diagonal(double *__restrict__ G, int n, int m)
{
    __shared__ double red[256];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) acc += G[(size_t)i * n + i];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    const double u = 1.1102230246251565e-16;  // 2^-53
    const double shift = 11.0 * ((double)m * n + (double)n * (n + 1)) * u * red[0];
    for (int i = threadIdx.x; i < n; i += blockDim.x) G[(size_t)i * n + i] += shift;
}

// Cholesky of the kb x kb diagonal block at (k0, k0) of the lower triangle of
// G (column-major, ld = n) into the same block of Lm, and the inverse of that
// factor into Linv (column-major, ld = kNb).  The block is padded to kNb x kNb
// with the identity.
//
// The factor is computed as G = L D L^T (L unit lower) by eliminating the
// augmented block [G | I], which leaves L^{-1} in the right half; the square
// roots come last (Cholesky factor L sqrt(D), inverse D^{-1/2} L^{-1}).  Panels
// of 8 columns, both halves in shared memory:
//   * warps 0-1 (a thread per row) and 2-3 (a thread per column of the right
//     half) each eliminate the panel's 8 x 8 diagonal block in registers,
//     carrying their own row or column along: nothing is exchanged on the chain
//     of pivots (a reciprocal and two fused operations each);
//   * warps 4-11 meanwhile subtract the previous panel's contribution from the
//     8 x 8 tiles that later panels need (two DMMA per tile), and scale and
//     write that panel's columns and rows;
//   * then warps 4-11 bring the next panel's tiles up to date, one tile each.
// Two barriers per panel.  What bounds it is the chain: 8 pivots per panel, 8
// panels.  Per block (B200, back to back): 49 us with one warp on each panel's
// chain and a division of labour by index arithmetic, 22.6 us with one or two
// columns per step spread over all threads (shared-memory loads and the
// step's exchange: 560 cycles per column), 18.5 with the tiles in registers
// (finding the next panel's among them: 1100 cycles per panel), 14.3 now.
// status <- 1 on a pivot that is not positive and finite.
constexpr int kDiagThreads = 384;

// 1 / d for a pivot d.  A pivot outside the approximation's range is divided
// by; one that is not positive and finite is replaced by 1 and clears ok.
__device__ __noinline__ double pc_reciprocal_rare(double &d, bool &ok)
{
    if (!(d > 0.0 && d < INFINITY)) {
        ok = false;
        d = 1.0;
    }
    return 1.0 / d;
}

__device__ __forceinline__ double pc_reciprocal(double &d, bool &ok)
{
    double r = approx_reciprocal(d);
    if (!reciprocal_in_range(d)) r = pc_reciprocal_rare(d, ok);
    return r;
}

constexpr int kDiagP = 8;                // columns per panel
constexpr int kDiagM = kNb + 2;          // row stride of the halves (16-byte row reads without bank conflicts)
constexpr int kDiagL = 12, kDiagX = kNb + 4;  // row strides of the panel's buffers (DMMA fragment reads likewise)
constexpr size_t kDiagSmem =
    sizeof(double) * (2 * kNb * kDiagM + 4 * kNb * kDiagL + 2 * kDiagP * kDiagX + 2 * kDiagP);

__global__ void __launch_bounds__(kDiagThreads, 1) pc_chol_inv_diag(const double *__restrict__ G,
                                                                    double *__restrict__ Lm, int n, int k0, int kb,
                                                                    double *__restrict__ Linv,
                                                                    int *__restrict__ status)
{
    constexpr int kP = kDiagP, kPanels = kNb / kP;
    extern __shared__ __align__(16) double dsm[];
    double(*A)[kDiagM] = reinterpret_cast<double(*)[kDiagM]>(dsm);  // left half (lower tiles), right half
    double(*X)[kDiagM] = A + kNb;
    double(*lp)[kNb][kDiagL] = reinterpret_cast<double(*)[kNb][kDiagL]>(X + kNb);  // L of the panel, by its parity
    double(*ld)[kNb][kDiagL] = lp + 2;                                             // L D of the panel
    double(*xo)[kP][kDiagX] = reinterpret_cast<double(*)[kP][kDiagX]>(ld + 2);     // its rows of L^{-1}
    double(*dv)[kP] = reinterpret_cast<double(*)[kP]>(xo + 2);                     // its pivots
    __shared__ double sq[kP], isq[kP];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    {
        constexpr int kIt = (kNb * kNb + kDiagThreads - 1) / kDiagThreads;
        double g[kIt];
#pragma unroll
        for (int u = 0; u < kIt; ++u) {
            const int e = t + u * kDiagThreads, i = e & (kNb - 1), k = e >> 6;
            g[u] = (i < kb && k < kb) ? (i >= k ? G[(size_t)(k0 + k) * n + k0 + i] : 0.0) : (i == k ? 1.0 : 0.0);
        }
#pragma unroll
        for (int u = 0; u < kIt; ++u) {
            const int e = t + u * kDiagThreads, i = e & (kNb - 1), k = e >> 6;
            if (e < kNb * kNb) {
                A[i][k] = g[u];
                X[i][k] = i == k ? 1.0 : 0.0;
            }
        }
    }
    __syncthreads();
    if (warp < 4) {
        const bool rows = warp < 2;
        const int i = t & (kNb - 1);
        for (int p = 0; p < kPanels; ++p) {
            const int b = p & 1, j0 = kP * p;
            // the diagonal block (lower triangle) and this thread's row of the
            // panel (warps 0-1) or column of the right half (warps 2-3)
            double d8[kP][kP], v[kP];
#pragma unroll
            for (int r = 0; r < kP; ++r)
#pragma unroll
                for (int q = 0; q <= r; q += 2) {
                    const double2 w = *reinterpret_cast<const double2 *>(&A[j0 + r][j0 + q]);
                    d8[r][q] = w.x;
                    if (q + 1 <= r) d8[r][q + 1] = w.y;
                }
            if (rows) {
#pragma unroll
                for (int j = 0; j < kP; j += 2) {
                    const double2 w = *reinterpret_cast<const double2 *>(&A[i][j0 + j]);
                    v[j] = w.x;
                    v[j + 1] = w.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < kP; ++j) v[j] = X[j0 + j][i];
            }
            double *lrow = lp[b][i], *drow = ld[b][i];
            bool ok = true;
#pragma unroll
            for (int j = 0; j < kP; ++j) {
                double d = d8[j][j];
                const double rd = pc_reciprocal(d, ok);
                if (t == 0) dv[b][j] = d;
                double l[kP];
#pragma unroll
                for (int r = j + 1; r < kP; ++r) {
                    l[r] = d8[r][j] * rd;
#pragma unroll
                    for (int q = j + 1; q <= r; ++q) d8[r][q] = fma(-l[r], d8[q][j], d8[r][q]);
                }
                if (rows) {
                    const double lv = v[j] * rd;
                    drow[j] = v[j];
                    lrow[j] = i > j0 + j ? lv : 0.0;
#pragma unroll
                    for (int q = j + 1; q < kP; ++q) v[q] = fma(-lv, d8[q][j], v[q]);
                } else {
#pragma unroll
                    for (int r = j + 1; r < kP; ++r) v[r] = fma(-l[r], v[j], v[r]);
                }
            }
            if (!rows) {
#pragma unroll
                for (int j = 0; j < kP; ++j) xo[b][j][i] = v[j];
            }
            if (t == 0 && !ok) atomicExch(status, 1);
            __syncthreads();                       // the panel is eliminated
            if (p + 1 < kPanels) __syncthreads();  // the next one is up to date
        }
    } else {
        const int fr = lane >> 2, fk = lane & 3, s = t - 128, w = warp - 4;
        // tile (i, c) of one half less panel p's contribution
        auto update = [&](int p, int i, int c, bool right) {
            const int b = p & 1;
            double2 *C = reinterpret_cast<double2 *>(right ? &X[8 * i + fr][8 * c + 2 * fk]
                                                           : &A[8 * i + fr][8 * c + 2 * fk]);
            const double *l = lp[b][8 * i + fr];
            const double a0 = -l[fk], a1 = -l[4 + fk];
            const double b0 = right ? xo[b][fk][8 * c + fr] : ld[b][8 * c + fr][fk];
            const double b1 = right ? xo[b][4 + fk][8 * c + fr] : ld[b][8 * c + fr][4 + fk];
            const double2 old = *C;
            double acc[2] = {old.x, old.y};
            dmma_m8n8k4(acc, a0, b0);
            dmma_m8n8k4(acc, a1, b1);
            *C = make_double2(acc[0], acc[1]);
        };
        // panel p's columns of the factor and rows of the inverse
        auto write_out = [&](int p) {
            const int b = p & 1;
            if (s < kP) {
                const double r = sqrt(dv[b][s]);
                sq[s] = r;
                isq[s] = 1.0 / r;
            }
            group_barrier(1, kDiagThreads - 128);
            for (int e = s; e < kP * kNb; e += kDiagThreads - 128) {
                const int i = e & (kNb - 1), j = e >> 6, k = kP * p + j;  // L(i, k)
                if (i >= k && i < kb) Lm[(size_t)(k0 + k) * n + k0 + i] = (i == k) ? sq[j] : lp[b][i][j] * sq[j];
                const int r = e & (kP - 1), c = e >> 3, row = kP * p + r;  // L^{-1}(row, c)
                Linv[row + (size_t)c * kNb] = (row < kb && c <= row) ? xo[b][r][c] * isq[r] : 0.0;
            }
        };
        for (int p = 0; p < kPanels; ++p) {
            if (p > 0) {
                // panel p - 1's contribution to the rows below panel p: left
                // half columns right of p, right half columns up to p - 1 (the
                // others' rows of L^{-1} are zero)
                int e = w;
                for (int i = p + 1; i < kPanels; ++i) {
                    const int left = i - p;
                    for (; e < left + p; e += 8) {
                        const bool right = e >= left;
                        update(p - 1, i, right ? e - left : p + 1 + e, right);
                    }
                    e -= left + p;
                }
                write_out(p - 1);
            }
            __syncthreads();
            if (p + 1 < kPanels) {
                // the next panel: left half rows p + 1 .. 7 of its column,
                // right half columns 0 .. p of its row
                const bool right = w > 6 - p;
                update(p, right ? p + 1 : p + 1 + w, right ? w - (7 - p) : p + 1, right);
                __syncthreads();
            }
        }
        write_out(kPanels - 1);
    }
}

// R (upper, column-major n x n) = L^T with zeros below the diagonal.
__global__ void pc_lower_to_upper(const double *__restrict__ L, double *__restrict__ R, int n)
{
    const size_t total = (size_t)n * n;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t i = e % n, j = e / n;  // R(i, j)
        R[e] = (i <= j) ? L[i * n + j] : 0.0;
    }
}

// One Cholesky QR pass: G = Q^T Q (+ shift), G = L L^T (blocked,
// right-looking; diagonal blocks factored and inverted by pc_chol_inv_diag,
// panels L21 = G21 L11^{-T} and trailing updates as GEMMs), then
// Qout = Q L^{-T} by a blocked right-looking solve (Qout_J = Q_J Linv_J^T,
// Q_{>J} -= Qout_J L_{>J,J}^T; Q is overwritten) and R = L^T.
int chol_qr_pass(cudaStream_t st, double *Q, double *Qout, int m, int n, double *G, double *Lm, double *Linv,
                 double *R, bool shift, int *d_status)
{
    JSVD_GEMM_TRY(dgemm(st, 'T', 'N', n, n, m, 1.0, Q, m, Q, m, 0.0, G, n, kGemmGram));
    if (shift) {
        pc_shift_diagonal<<<1, 256, 0, st>>>(G, n, m);
        JSVD_CUDA_TRY(cudaGetLastError());
    }
    for (int k0 = 0, blk = 0; k0 < n; k0 += kNb, ++blk) {
        const int kb = std::min(kNb, n - k0);
        double *li = Linv + (size_t)blk * kNb * kNb;
        pc_chol_inv_diag<<<1, kDiagThreads, kDiagSmem, st>>>(G, Lm, n, k0, kb, li, d_status);
        JSVD_CUDA_TRY(cudaGetLastError());
        const int rest = n - k0 - kb;
        if (rest > 0) {
            // L21 = G21 L11^{-T}
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', rest, kb, kb, 1.0, G + (size_t)k0 * n + k0 + kb, n, li, kNb, 0.0,
                                Lm + (size_t)k0 * n + k0 + kb, n));
            // G22 -= L21 L21^T (lower)
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', rest, rest, kb, -1.0, Lm + (size_t)k0 * n + k0 + kb, n,
                                Lm + (size_t)k0 * n + k0 + kb, n, 1.0, G + (size_t)(k0 + kb) * n + k0 + kb, n,
                                kGemmLower));
        }
    }
    for (int j0 = 0, blk = 0; j0 < n; j0 += kNb, ++blk) {
        const int kb = std::min(kNb, n - j0);
        const double *li = Linv + (size_t)blk * kNb * kNb;
        JSVD_GEMM_TRY(
            dgemm(st, 'N', 'T', m, kb, kb, 1.0, Q + (size_t)j0 * m, m, li, kNb, 0.0, Qout + (size_t)j0 * m, m));
        const int rest = n - j0 - kb;
        if (rest > 0)
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', m, rest, kb, -1.0, Qout + (size_t)j0 * m, m, Lm + (size_t)j0 * n + j0 + kb,
                                n, 1.0, Q + (size_t)(j0 + kb) * m, m));
    }
    pc_lower_to_upper<<<std::min<size_t>(1184, ((size_t)n * n + 255) / 256), 256, 0, st>>>(Lm, R, n);
    JSVD_CUDA_TRY(cudaGetLastError());
    return JSVD_OK;
}

std::atomic<int> g_inner{1};
std::atomic<int> g_gram_stop{1};

// The Jacobi stage on X (row-major cols x cols): the plain sweep (default) or,
// when selected, the block-pair engine where it applies.  The plain sweep
// measured faster on B200 for the 1024-column factor of a 4096 x 1024 input
// (2.6 us per round, 1023 rounds per sweep, against 18 us per block-pair outer
// round, 255 per sweep).
// Engine 2 is the blocked mixed-precision sweep (mixed.cu), used by
// jsvd_mixed_svd*.
constexpr int kEngineMixed = 2;

int inner_jacobi(const double *x, size_t cols, const jsvd_config &c, double *u, double *sigma, double *v, int *sweeps,
                 cudaStream_t st, int engine)
{
    if (engine == kEngineMixed && cols >= (size_t)kMixedMinCols)
        return mixed_solve(x, (int)cols, (int)cols, c, mixed_options(), u, sigma, v, sweeps, st);
    if (engine == 0 && bp_supported(cols, cols))
        return bp_solve(x, cols, cols, c.epsilon, c.max_sweeps, u, sigma, v, sweeps, st);
    // The last, rotation-free sweep is replaced by a test of every pair on the
    // Gram matrix (this path is held to a tolerance, not to the bits).
    return plain_device_solve(x, cols, cols, &c, u, sigma, v, sweeps, st, g_gram_stop.load() != 0);
}

struct PrecondStats {
    unsigned long long solves = 0, fallbacks = 0;
    double qr_ms = 0.0, jacobi_ms = 0.0, u_ms = 0.0;
    int last_sweeps = 0;
};

PrecondStats &precond_stats()
{
    thread_local PrecondStats s;
    return s;
}

// Per-thread cached resources of the QR stage for one shape: the workspace,
// a stream for allocation and graph capture, and the two shifted CholeskyQR3
// stages captured as graphs on the plan's second use.  The stage is ~500 small
// launches whose enqueueing, not their device time, set its duration.
struct PcPlan {
    int device = -1;
    size_t m = 0, n = 0;
    double *ws = nullptr;
    cudaStream_t own = nullptr;
    cudaGraphExec_t qr1 = nullptr, qr2 = nullptr;
    bool no_graph = false;  // a capture failed: launch directly from then on
    unsigned long long uses = 0;
    ~PcPlan()
    {
        if (qr1) cudaGraphExecDestroy(qr1);
        if (qr2) cudaGraphExecDestroy(qr2);
        if (own) {
            if (ws) cudaFreeAsync(ws, own);
            cudaStreamSynchronize(own);
            cudaStreamDestroy(own);
        }
    }
};

constexpr size_t kPcMaxPlanBytes = size_t(2) << 30;  // larger shapes allocate per call, no graphs
constexpr size_t kPcMaxPlans = 2;

std::vector<std::unique_ptr<PcPlan>> &pc_plans()
{
    thread_local std::vector<std::unique_ptr<PcPlan>> plans;
    return plans;
}

// The cached plan for (device, m, n), created on first use; nullptr (and
// JSVD_OK) when the shape's workspace is above kPcMaxPlanBytes.
int acquire_pc_plan(int dev, size_t m, size_t n, size_t ws_doubles, PcPlan **out)
{
    *out = nullptr;
    if (sizeof(double) * ws_doubles > kPcMaxPlanBytes) return JSVD_OK;
    auto &plans = pc_plans();
    for (size_t i = 0; i < plans.size(); ++i) {
        if (plans[i]->device == dev && plans[i]->m == m && plans[i]->n == n) {
            std::rotate(plans.begin(), plans.begin() + i, plans.begin() + i + 1);
            *out = plans.front().get();
            return JSVD_OK;
        }
    }
    auto p = std::make_unique<PcPlan>();
    p->device = dev;
    p->m = m;
    p->n = n;
    {
        const cudaError_t e = cudaStreamCreateWithFlags(&p->own, cudaStreamNonBlocking);
        if (e != cudaSuccess) {
            p->own = nullptr;
            return cuda_failure(e, "cudaStreamCreateWithFlags", __FILE__, __LINE__);
        }
    }
    JSVD_CUDA_TRY(cudaMallocAsync((void **)&p->ws, sizeof(double) * ws_doubles, p->own));
    JSVD_CUDA_TRY(cudaStreamSynchronize(p->own));
    plans.insert(plans.begin(), std::move(p));
    while (plans.size() > kPcMaxPlans) plans.pop_back();
    *out = plans.front().get();
    return JSVD_OK;
}

int precond_impl(const double *d_a, size_t rows, size_t cols, const jsvd_config &c, double *d_u, double *d_sigma,
                 double *d_v, int *sweeps, cudaStream_t st, int engine)
{
    const int m = (int)rows, n = (int)cols;
    int dev = 0;
    JSVD_CUDA_TRY(cudaGetDevice(&dev));
    const size_t mn = (size_t)m * n, nn = (size_t)n * n;
    // workspace: Qa, Qb (m x n) | G | Lm | R1 | R2 | R3 | T | Vx | Ux | Sa | Sb | P1 (n x n)
    //            | Linv (blocks x 64 x 64) | sigma | status
    const int nblk = (n + kNb - 1) / kNb;
    const size_t ws_doubles = 2 * mn + 11 * nn + (size_t)nblk * kNb * kNb + n + 1;
    PcPlan *plan = nullptr;
    int rc = acquire_pc_plan(dev, rows, cols, ws_doubles, &plan);
    if (rc != JSVD_OK) return rc;
    JSVD_CUDA_TRY(cudaFuncSetAttribute(pc_chol_inv_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiagSmem));
    double *ws = plan ? plan->ws : nullptr;
    if (!plan) JSVD_CUDA_TRY(cudaMallocAsync((void **)&ws, sizeof(double) * ws_doubles, st));
    double *Qa = ws, *Qb = Qa + mn, *G = Qb + mn, *Lm = G + nn, *R1 = Lm + nn, *R2 = R1 + nn, *R3 = R2 + nn,
           *Tm = R3 + nn, *Vx = Tm + nn, *Ux = Vx + nn, *Sa = Ux + nn, *Sb = Sa + nn, *P1 = Sb + nn,
           *Linv = P1 + nn, *sg = Linv + (size_t)nblk * kNb * kNb;
    int *d_status = reinterpret_cast<int *>(sg + n);
    double *Q = Qb;   // after three passes (Qa -> Qb -> Qa -> Qb) the factor is in Qb
    double *Q1 = Sb;  // likewise for the second factorisation (Sa -> Sb -> Sa -> Sb)
    cudaEvent_t e0, e1, e2, e3;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventCreate(&e2);
    cudaEventCreate(&e3);
    bool cleaned = false;
    auto cleanup = [&]() {
        if (cleaned) return;
        cleaned = true;
        if (!plan) cudaFreeAsync(ws, st);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        cudaEventDestroy(e2);
        cudaEventDestroy(e3);
    };
    // every return below, the early ones of the status macros included, releases them
    ScopeExit guard([&] { cleanup(); });
    // Shifted CholeskyQR3 of Xa (rows x n, column-major, overwritten): the
    // orthonormal factor ends in Xb, R = R3 R2 R1 in Ra (upper, column-major);
    // Rb, Rc are scratch.
    auto scqr3 = [&](cudaStream_t s2, double *Xa, double *Xb, int rows, double *Ra, double *Rb, double *Rc) -> int {
        int r = chol_qr_pass(s2, Xa, Xb, rows, n, G, Lm, Linv, Ra, true, d_status);
        if (r == JSVD_OK) r = chol_qr_pass(s2, Xb, Xa, rows, n, G, Lm, Linv, Rb, false, d_status);
        if (r == JSVD_OK) r = chol_qr_pass(s2, Xa, Xb, rows, n, G, Lm, Linv, Rc, false, d_status);
        if (r != JSVD_OK) return r;
        JSVD_GEMM_TRY(dgemm(s2, 'N', 'N', n, n, n, 1.0, Rb, n, Ra, n, 0.0, Tm, n, kGemmUpper));
        JSVD_GEMM_TRY(dgemm(s2, 'N', 'N', n, n, n, 1.0, Rc, n, Tm, n, 0.0, Ra, n, kGemmUpper));
        return JSVD_OK;
    };
    // Runs a QR stage: directly, or (a plan on its second use onwards) as a
    // graph captured once on the plan's own stream and replayed on st.
    auto run_stage = [&](cudaGraphExec_t *exec, auto &&enqueue) -> int {
        if (plan && !plan->no_graph && *exec == nullptr && plan->uses >= 1) {
            cudaGraph_t graph = nullptr;
            int r = JSVD_OK;
            cudaError_t ce = cudaStreamBeginCapture(plan->own, cudaStreamCaptureModeThreadLocal);
            if (ce == cudaSuccess) {
                r = enqueue(plan->own);
                ce = cudaStreamEndCapture(plan->own, &graph);
            }
            if (r == JSVD_OK && ce == cudaSuccess && graph != nullptr) {
                if (cudaGraphInstantiate(exec, graph, 0) != cudaSuccess) *exec = nullptr;
            }
            if (graph) cudaGraphDestroy(graph);
            if (*exec == nullptr) {
                plan->no_graph = true;  // launch directly from now on
                cudaGetLastError();
                set_last_error(JSVD_OK, "");
            }
        }
        if (plan && *exec != nullptr) {
            JSVD_CUDA_TRY(cudaGraphLaunch(*exec, st));
            return JSVD_OK;
        }
        return enqueue(st);
    };
    auto read_status = [&](int *out) -> int {
        JSVD_CUDA_TRY(cudaMemcpyAsync(out, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
        JSVD_CUDA_TRY(cudaStreamSynchronize(st));
        return JSVD_OK;
    };
    cudaEventRecord(e0, st);
    JSVD_CUDA_TRY(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    JSVD_CUDA_TRY(launch_rowmajor_to_colmajor(d_a, m, n, Qa, m, st));
    // A = Q R
    rc = run_stage(plan ? &plan->qr1 : nullptr,
                   [&](cudaStream_t s2) { return scqr3(s2, Qa, Qb, m, R1, R2, R3); });
    int status = 0;
    if (rc == JSVD_OK) rc = read_status(&status);
    if (rc != JSVD_OK) {
        cleanup();
        return rc;
    }
    PrecondStats &ps = precond_stats();
    if (status != 0) {
        // Gram not positive definite in floating point: plain path on A.
        cudaEventRecord(e1, st);
        cleanup();
        ps.fallbacks += 1;
        if (engine == kEngineMixed) mixed_note_solve(0.0, true);
        return jsvd_plain_svd_device(d_a, rows, cols, &c, d_u, d_sigma, d_v, sweeps, st);
    }
    // R^T = Q1 P (P upper): R1's column-major buffer read as row-major is R^T.
    rc = run_stage(plan ? &plan->qr2 : nullptr, [&](cudaStream_t s2) -> int {
        pc_to_colmajor<<<dim3((n + kTile - 1) / kTile, (n + kTile - 1) / kTile), dim3(kTile, kTileRows), 0, s2>>>(
            R1, n, n, Sa);
        JSVD_CUDA_TRY(cudaGetLastError());
        return scqr3(s2, Sa, Sb, n, P1, R2, R3);
    });
    int status2 = 0;
    if (rc == JSVD_OK) rc = read_status(&status2);
    if (rc != JSVD_OK) {
        cleanup();
        return rc;
    }
    cudaEventRecord(e1, st);
    double *sout = d_sigma ? d_sigma : sg;
    if (status2 == 0) {
        // A = Q R = Q P^T Q1^T.  Jacobi on X = P^T (P1's column-major buffer read
        // as row-major): X = Ux S Vx^T, so U_A = Q Ux and V_A = Q1 Vx.
        rc = inner_jacobi(P1, cols, c, d_u ? Ux : nullptr, sout, d_v ? Vx : nullptr, sweeps, st, engine);
        if (rc != JSVD_OK) {
            cleanup();
            return rc;
        }
        cudaEventRecord(e2, st);
        // Row-major U_A (m x n) is column-major U_A^T = Ux^T Q^T; Ux's row-major
        // buffer is Ux^T column-major.  The same for V_A^T = Vx^T Q1^T.
        if (d_u)
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', n, m, n, 1.0, Ux, n, Q, m, 0.0, d_u, n));
        if (d_v)
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', n, n, n, 1.0, Vx, n, Q1, n, 0.0, d_v, n));
    } else {
        // Second factorisation failed: Jacobi on X = R^T, A = Q X^T =
        // (Q Vx) S Ux^T, so U_A = Q Vx and V_A = Ux.
        ps.fallbacks += 1;
        double *vout = d_v ? d_v : Ux;
        rc = inner_jacobi(R1, cols, c, vout, sout, Vx, sweeps, st, engine);
        if (rc != JSVD_OK) {
            cleanup();
            return rc;
        }
        cudaEventRecord(e2, st);
        if (d_u)
            JSVD_GEMM_TRY(dgemm(st, 'N', 'T', n, m, n, 1.0, Vx, n, Q, m, 0.0, d_u, n));
    }
    cudaEventRecord(e3, st);
    JSVD_CUDA_TRY(cudaStreamSynchronize(st));
    float a = 0, b = 0, d = 0;
    cudaEventElapsedTime(&a, e0, e1);
    cudaEventElapsedTime(&b, e1, e2);
    cudaEventElapsedTime(&d, e2, e3);
    ps.solves += 1;
    ps.qr_ms += a;
    ps.jacobi_ms += b;
    ps.u_ms += d;
    ps.last_sweeps = sweeps ? *sweeps : 0;
    if (engine == kEngineMixed) mixed_note_solve(a, status2 != 0);
    if (plan) plan->uses += 1;
    cleanup();
    return JSVD_OK;
}

}  // namespace
}  // namespace jsvd

using namespace jsvd;

extern "C" int jsvd_precond_svd_device(const double *d_a, size_t rows, size_t columns, const jsvd_config *cfg,
                                       double *d_u, double *d_sigma, double *d_v, int *sweeps, void *stream)
{
    return c_entry([&]() -> int {
        set_last_error(JSVD_OK, "");
        jsvd_config def;
        const jsvd_config &c = config_or_default(cfg, def);
        int rc = validate_plain_request(d_a, rows, columns, c);
        if (rc != JSVD_OK) return rc;
        cudaStream_t st = nullptr;
        if (const int e = entry_stream(stream, &st); e != JSVD_OK) return e;
        if (columns == 1) return jsvd_plain_svd_device(d_a, rows, columns, &c, d_u, d_sigma, d_v, sweeps, st);
        return precond_impl(d_a, rows, columns, c, d_u, d_sigma, d_v, sweeps, st, g_inner.load());
    });
}

extern "C" int jsvd_precond_svd(const double *a, size_t rows, size_t columns, const jsvd_config *cfg, double *u,
                                double *sigma, double *v, int *sweeps)
{
    return c_entry([&]() -> int {
        return host_buffer_solve(jsvd_precond_svd_device, a, rows, columns, cfg, u, sigma, v, sweeps);
    });
}

namespace jsvd {
void pc_release_thread_plans() { pc_plans().clear(); }
}  // namespace jsvd

extern "C" int jsvd_mixed_svd_device(const double *d_a, size_t rows, size_t columns, const jsvd_config *cfg,
                                     double *d_u, double *d_sigma, double *d_v, int *sweeps, void *stream)
{
    return c_entry([&]() -> int {
        set_last_error(JSVD_OK, "");
        jsvd_config def;
        const jsvd_config &c = config_or_default(cfg, def);
        int rc = validate_plain_request(d_a, rows, columns, c);
        if (rc != JSVD_OK) return rc;
        cudaStream_t st = nullptr;
        if (const int e = entry_stream(stream, &st); e != JSVD_OK) return e;
        if (columns == 1) return jsvd_plain_svd_device(d_a, rows, columns, &c, d_u, d_sigma, d_v, sweeps, st);
        const jsvd_mixed_options &o = mixed_options();
        if (!o.precondition && columns >= (size_t)kMixedMinCols) {
            // the blocked sweeps directly on A (row tiles of 32 along the
            // transpose grid's y dimension bound the rows)
            if (rows > (size_t)65535 * 32)
                return invalid_argument("jsvd_mixed_svd: too many rows for the unpreconditioned blocked sweep.");
            rc = mixed_solve(d_a, (int)rows, (int)columns, c, o, d_u, d_sigma, d_v, sweeps, st);
            if (rc == JSVD_OK) mixed_note_solve(0.0, false);
            return rc;
        }
        return precond_impl(d_a, rows, columns, c, d_u, d_sigma, d_v, sweeps, st, kEngineMixed);
    });
}

extern "C" int jsvd_mixed_svd(const double *a, size_t rows, size_t columns, const jsvd_config *cfg, double *u,
                              double *sigma, double *v, int *sweeps)
{
    return c_entry([&]() -> int {
        return host_buffer_solve(jsvd_mixed_svd_device, a, rows, columns, cfg, u, sigma, v, sweeps);
    });
}

extern "C" void jsvd_precond_set_inner(int engine) { g_inner.store(engine == 0 ? 0 : 1); }

extern "C" void jsvd_precond_set_gram_stop(int enable) { g_gram_stop.store(enable ? 1 : 0); }

extern "C" void jsvd_precond_stats_get(jsvd_precond_stats *out)
{
    if (!out) return;
    const PrecondStats &s = precond_stats();
    out->solves = s.solves;
    out->fallbacks = s.fallbacks;
    out->qr_ms = s.qr_ms;
    out->jacobi_ms = s.jacobi_ms;
    out->u_ms = s.u_ms;
}

extern "C" void jsvd_precond_stats_reset(void) { precond_stats() = PrecondStats{}; }
