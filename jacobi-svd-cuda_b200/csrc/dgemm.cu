// FP64 GEMM for sm_100a on the FP64 tensor cores.
//
// tcgen05 has no FP64 kind, so the FP64 products of this library (CholeskyQR
// Grams and triangular updates, re-orthogonalisation, U = Q U_x, V = Q1 V_x)
// run on mma.sync m8n8k4 f64 (DMMA).  Each warp owns a 32 x 32 tile of C (16
// DMMA tiles, 32 accumulators per lane); a CTA of 4 warps owns 64 x 64, two or
// three CTAs to an SM (three_ctas), so that one's loads, barriers and epilogue
// pass under the other's DMMA.  Measured against one 128 x 128 CTA of 16 warps
// (B200): 4096^3 op T,N 4.42 ms, 31.1 TFLOP/s (4.93, 27.9); 1024 x 8192 x 1024 op
// N,T 0.590 ms (0.778); 128 x 64 lies between (4.70, 0.692).  Operand tiles of
// BK = 16 are staged in shared memory through a 3-stage cp.async ring.
// Every operand is stored in shared memory along the dimension that is
// contiguous in global memory, so global reads are coalesced and shared-memory
// writes conflict-free:
//   MN-contiguous [k][mn] (row length 64 + 8: fragment reads of 8 x 4 doubles
//     take the minimum two wavefronts) for op(A) = N and op(B) = T;
//   K-contiguous  [mn][k] (row length BK + 4, same property) for op(A) = T and
//     op(B) = N.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "dgemm.hpp"
#include "internal.hpp"
#include "jsvd.h"
#include "plain.hpp"
#include "ptx.cuh"

namespace jsvd {
namespace {

namespace cg = cooperative_groups;

constexpr int kBM = 64, kBN = 64;  // tile of C per CTA
constexpr int kThreads = (kBM / 32) * (kBN / 32) * 32;
constexpr int kBK = 16;
constexpr int kStages = 3;

template <bool KCONTIG, int BMN>
struct OperandTile {
    // elements per stage, row length
    static constexpr int LD = KCONTIG ? (kBK + 4) : (BMN + 8);
    static constexpr int ELEMS = KCONTIG ? BMN * LD : kBK * LD;
    __device__ static int idx(int mn, int k) { return KCONTIG ? mn * LD + k : k * LD + mn; }
};

// Loads the kBK-deep slice k0 of op(X) rows [mn0, mn0 + BMN) into s.  X is
// column-major with leading dimension ldx.  For op = N of A (and op = T of B)
// the contiguous global dimension is mn; otherwise it is k.
template <bool KCONTIG, int BMN>
__device__ __forceinline__ void load_tile(double *s, const double *X, long ldx, int mn0, int k0, int MN, int K)
{
    using Tl = OperandTile<KCONTIG, BMN>;
    constexpr int TOTAL = BMN * kBK;
#pragma unroll
    for (int e0 = 0; e0 < TOTAL; e0 += kThreads) {
        const int e = e0 + (int)threadIdx.x;
        int mn, k;
        if (KCONTIG) {
            k = e % kBK;
            mn = e / kBK;
        } else {
            mn = e % BMN;
            k = e / BMN;
        }
        const int gm = mn0 + mn, gk = k0 + k;
        double *dst = s + Tl::idx(mn, k);
        if (gm < MN && gk < K) {
            // KCONTIG: X(k, mn) at k + mn*ldx;  MN-contiguous: X(mn, k) at mn + k*ldx
            const double *src = KCONTIG ? (X + (size_t)gk + (size_t)gm * ldx) : (X + (size_t)gm + (size_t)gk * ldx);
            cp_async8(dst, src);
        } else {
            *dst = 0.0;
        }
    }
}

// kForm: the forms with a triangle have kernels of their own, because their
// bounds in the general one cost it 6 % (168 registers for 202).  kBeta: with
// three CTAs to an SM, whose registers are the tighter ones, beta = 0 has a
// kernel without C's old values (1 to 2 %); otherwise it is decided at run time.
template <bool TA, bool TB, GemmForm kForm, int kCtas, bool kBeta>
__global__ void __launch_bounds__(kThreads, kCtas)
    dgemm_kernel(int m, int n, int k, double alpha, const double *__restrict__ A, long lda,
                 const double *__restrict__ B, long ldb, double beta, double *__restrict__ C, long ldc, int lower)
{
    constexpr int WN = kBN / 32;
    // op(A) = N: A(m x k) contiguous along m -> MN-contiguous; op(A) = T: K-contiguous.
    // op(B) = N: B(k x n) contiguous along k -> K-contiguous;  op(B) = T: MN-contiguous.
    constexpr bool AK = TA, BKc = !TB;
    using TA_ = OperandTile<AK, kBM>;
    using TB_ = OperandTile<BKc, kBN>;
    extern __shared__ double dsm[];
    double *sa = dsm;
    double *sb = dsm + kStages * TA_::ELEMS;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
    constexpr bool kSplit = kForm == kGemmGram;
    if ((kForm == kGemmSymmetric || kSplit || lower) && n0 > m0 + kBM - 1) return;  // tile strictly above the diagonal
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp / WN, wn = warp % WN;
    // Upper times upper: k in [m0, n0 + kBN), empty below the diagonal; the
    // terms left out are products with a zero.  1/6 of the full product's work.
    // With V^T V from its lower tiles, a mixed solve of 8192 x 4096: 425 -> 405
    // ms, of 1777 x 611: 12.83 -> 12.58 ms.
    int first = kForm == kGemmUpper ? m0 / kBK : 0;
    int last = ((kForm == kGemmUpper ? min(k, n0 + kBN) : k) + kBK - 1) / kBK;
    if constexpr (kSplit) {
        first = (int)((long)last * blockIdx.z / gridDim.z);
        last = (int)((long)last * (blockIdx.z + 1) / gridDim.z);
    }

    auto issue = [&](int kt) {
        const int s = kt % kStages;
        load_tile<AK, kBM>(sa + s * TA_::ELEMS, A, lda, m0, kt * kBK, m, k);
        load_tile<BKc, kBN>(sb + s * TB_::ELEMS, B, ldb, n0, kt * kBK, n, k);
    };

    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (first + s < last) issue(first + s);
        cp_async_commit();
    }
    const int fr = lane >> 2, fk = lane & 3;
    for (int kt = first; kt < last; ++kt) {
        cp_async_wait<kStages - 2>();
        __syncthreads();
        if (kt + kStages - 1 < last) issue(kt + kStages - 1);
        cp_async_commit();
        const double *ta = sa + (kt % kStages) * TA_::ELEMS;
        const double *tb = sb + (kt % kStages) * TB_::ELEMS;
#pragma unroll
        for (int kk = 0; kk < kBK; kk += 4) {
            double af[4], bf[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) af[i] = ta[TA_::idx(wm * 32 + i * 8 + fr, kk + fk)];
#pragma unroll
            for (int j = 0; j < 4; ++j) bf[j] = tb[TB_::idx(wn * 32 + j * 8 + fr, kk + fk)];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma_m8n8k4(acc[i][j], af[i], bf[j]);
        }
    }
    cp_async_wait<0>();
    if constexpr (kSplit) {
        // The cluster's CTAs hold parts of one tile: each leaves its part in
        // shared memory, then adds an equal share of the tile's columns over the
        // ranks, in their order.
        constexpr int kLd = kBM + 2;
        static_assert(kBN * kLd <= kStages * (TA_::ELEMS + TB_::ELEMS), "the part fits the staging buffers");
        cg::cluster_group cluster = cg::this_cluster();
        const int parts = (int)gridDim.z;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    dsm[(wn * 32 + j * 8 + 2 * fk + h) * kLd + wm * 32 + i * 8 + fr] = acc[i][j][h];
        cluster.sync();
        const int share = kBN / parts;
        for (int e = (int)threadIdx.x; e < share * kBM; e += kThreads) {
            const int c = (int)blockIdx.z * share + e / kBM, r = e % kBM;
            double sum = 0.0;
            for (int p = 0; p < parts; ++p) sum += cluster.map_shared_rank(dsm, p)[c * kLd + r];
            if (m0 + r < m && n0 + c < n && n0 + c <= m0 + r) C[(size_t)(m0 + r) + (size_t)(n0 + c) * ldc] = alpha * sum;
        }
        cluster.sync();  // no CTA leaves while another reads its part
        return;
    }
    // C's old values are all loaded before any store: a load cannot pass a
    // store to the same array, so one element at a time the epilogue was a chain
    // of 32 loads (a 64 x 64 x 64 product with beta = 1: 20 us, with beta = 0:
    // 7.6 us, alone on the device).
    double old[4][4][2];
    const bool add = kCtas == 2 ? beta != 0.0 : kBeta;
    if (add) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = m0 + wm * 32 + i * 8 + fr, col = n0 + wn * 32 + j * 8 + 2 * fk + h;
                    const bool live = row < m && col < n && !(lower && col > row);
                    old[i][j][h] = live ? C[(size_t)row + (size_t)col * ldc] : 0.0;
                }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = m0 + wm * 32 + i * 8 + fr;
        if (row >= m) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = n0 + wn * 32 + j * 8 + 2 * fk + h;
                if (col >= n || (lower && col > row)) continue;
                const double v = alpha * acc[i][j][h];
                C[(size_t)row + (size_t)col * ldc] = add ? fma(beta, old[i][j][h], v) : v;
                if (kForm == kGemmSymmetric && n0 < m0) C[(size_t)col + (size_t)row * ldc] = v;
            }
        }
    }
}

// lower: for kGemmGram the number of parts, else whether only the lower
// triangle is written
template <bool TA, bool TB, GemmForm kForm, int kCtas = 2, bool kBeta = true>
int launch(cudaStream_t st, int m, int n, int k, double alpha, const double *A, long lda, const double *B, long ldb,
           double beta, double *C, long ldc, int lower)
{
    constexpr size_t smem = sizeof(double) * kStages *
                            (OperandTile<TA, kBM>::ELEMS + OperandTile<!TB, kBN>::ELEMS);
    static_assert(smem <= 227 * 1024, "dgemm tile does not fit shared memory");
    auto kern = dgemm_kernel<TA, TB, kForm, kCtas, kBeta>;
    if (smem > 48 * 1024)
        JSVD_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((m + kBM - 1) / kBM, (n + kBN - 1) / kBN);
    if constexpr (kForm == kGemmGram) {
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim = {1, 1, (unsigned)lower};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid.x, grid.y, (unsigned)lower);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        JSVD_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, 1));
        return JSVD_OK;
    }
    kern<<<grid, kThreads, smem, st>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lower);
    JSVD_CUDA_TRY(cudaGetLastError());
    return JSVD_OK;
}

// SMs of the current device.
int device_sms()
{
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    if (dev < 64 && (sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
    if (dev < 64) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// Whether a product of `tiles` tiles runs three CTAs to an SM (168 registers) or
// two (202).  Two take the tiles of an SM in pairs, three in threes, and a short
// last wave costs nearly a whole one: with the tiles per SM rounded up, 512 x N x
// 1024 op N,N takes (us, B200, two / three)
//   1: 76 / 77   2: 99 / 101   3: 182 / 148   4: 183 / 225   5: 265 / 225
//   6: 265 / 269   7: 348 / 310   8: 348 / 347   9: 431 / 388   28: 1180 / 1150
// and lower triangles the same way (k = 2048, 300 tiles: 290 / 263, 528: 332 / 410).
bool three_ctas(long tiles)
{
    const int sms = device_sms();
    const long load = (tiles + sms - 1) / sms;
    return load >= 8 || load == 3 || load == 5 || load == 7;
}

// Parts of the sum over k of an n x n Gram: as many (a power of two, at most 8)
// as keep the tiles on and below the diagonal within two CTAs to an SM, each
// part at least 128 deep: unsplit, the 36 tiles of a 512-column Gram leave 112
// SMs idle and one warp per scheduler with nothing to hide its loads.  B200,
// QR-preconditioned solve of 2048 x 512 10.80 -> 10.53 ms, mixed 1777 x 611
// 12.58 -> 12.32.  The parts' shorter sums round less than the single one.
int gram_parts(int n, int k)
{
    const long t = (n + kBN - 1) / kBN, tiles = t * (t + 1) / 2;
    int parts = 1;
    while (parts < 8 && tiles * parts * 2 <= 2 * device_sms() && k / (parts * 2) >= 128) parts *= 2;
    return parts;
}

thread_local unsigned long long t_launches = 0;

}  // namespace

unsigned long long dgemm_launches() { return t_launches; }

int dgemm(cudaStream_t st, char opA, char opB, int m, int n, int k, double alpha, const double *A, long lda,
          const double *B, long ldb, double beta, double *C, long ldc, GemmForm form)
{
    if (m <= 0 || n <= 0) return JSVD_OK;
    if (k <= 0) return invalid_argument("dgemm: k must be positive.");
    if (m > 65535 * 64 || n > 65535 * 64) return invalid_argument("dgemm: matrix too large for the tile grid.");
    ++t_launches;
    const bool ta = (opA == 'T' || opA == 't'), tb = (opB == 'T' || opB == 't');
    if (form == kGemmGram) {
        if (!ta || tb || m != n || beta != 0.0)
            return invalid_argument("dgemm: the product does not have the form asked for.");
        const int parts = gram_parts(n, k);
        if (parts > 1)
            return launch<true, false, kGemmGram>(st, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, parts);
        form = kGemmLower;
    }
    const auto run = [&](auto of) { return of(st, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, form == kGemmLower); };
    if (form == kGemmSymmetric || form == kGemmUpper) {
        const bool upper = form == kGemmUpper;
        if (ta == upper || tb || m != n || (upper && k != n) || beta != 0.0)
            return invalid_argument("dgemm: the product does not have the form asked for.");
        return upper ? run(launch<false, false, kGemmUpper>) : run(launch<true, false, kGemmSymmetric>);
    }
    const long mt = (m + kBM - 1) / kBM, nt = (n + kBN - 1) / kBN, diagonal = std::min(mt, nt);
    const bool three = three_ctas(form == kGemmLower ? diagonal * mt - diagonal * (diagonal - 1) / 2 : mt * nt);
    const auto pick = [&](auto opa, auto opb) {
        constexpr bool A_ = decltype(opa)::value, B_ = decltype(opb)::value;
        if (!three) return run(launch<A_, B_, kGemmFull>);
        return beta != 0.0 ? run(launch<A_, B_, kGemmFull, 3, true>) : run(launch<A_, B_, kGemmFull, 3, false>);
    };
    const std::true_type T{};
    const std::false_type N{};
    if (!ta) return tb ? pick(N, T) : pick(N, N);
    return tb ? pick(T, T) : pick(T, N);
}

}  // namespace jsvd

// Test and tooling entry: C = alpha op(A) op(B) + beta C on device buffers,
// on the calling thread's library stream, synchronously.
extern "C" int jsvd_dgemm_device(char op_a, char op_b, int m, int n, int k, double alpha, const double *a, long lda,
                                 const double *b, long ldb, double beta, double *c, long ldc, int lower)
{
    using namespace jsvd;
    return c_entry([&]() -> int {
        set_last_error(JSVD_OK, "");
        if (!a || !b || !c) return invalid_argument("jsvd_dgemm_device: null buffer.");
        cudaStream_t st = nullptr;
        if (const int e = entry_stream(nullptr, &st); e != JSVD_OK) return e;
        const int rc = dgemm(st, op_a, op_b, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc,
                             lower ? kGemmLower : kGemmFull);
        if (rc != JSVD_OK) return rc;
        JSVD_CUDA_TRY(cudaStreamSynchronize(st));
        return JSVD_OK;
    });
}
