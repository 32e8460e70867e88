// Batched one-sided Jacobi SVD: thousands of independent small matrices,
// persistent launches per size class, largest class first (sm_100a).  A class's
// members are split by the kernel that suits them: the one-CTA kernel by a bound
// on their rows, clusters by their size.
//
// Each CTA pulls matrix indices from a device work queue (one atomic counter
// per launch; matrices sorted by work, largest first) and solves the whole
// matrix before taking the next one.  Where the FP64 working copies live
// depends on the class:
//   class 0-2: A and V in shared memory (<= 48 KiB, <= 100 KiB, <= ~226 KiB)
//   class 3  : A in shared memory, V in a per-CTA slice of global memory
//   class 4  : A and V in global memory (L2-resident per-CTA slices), the
//              leading columns of A that fit in shared memory kept there
// By default the members of class 4, and of class 3 while they are few, are
// instead solved by a thread-block cluster each (batch_cluster_kernel: A and V in
// the cluster's distributed shared memory; see the section "cluster classes"); a
// member no cluster holds stays with its class's kernel.
// Launch shapes per class (threads, CTAs per SM, grid cap) come from the
// compiled-in table batch_tuning_table.h, which batch_autotune.py writes from
// jsvd_batch_autotune (defined at the end of this file).
// Each round runs in three phases separated by __syncthreads:
//   1. one warp per pair: the three dot products, reduced in the reference's
//      order (T = 256 virtual lanes; lane l holds virtual lanes l + 32j, then
//      the halving tree) - so every matrix is bit-identical to the plain path
//      and to the oracle on the same (FP64-promoted) input;
//   2. one thread per pair: the rotation angle (the long sqrt/div chain runs
//      for all pairs of the round in parallel instead of serially per warp);
//   3. one warp per pair: rotation of the A and V columns.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <numeric>
#include <queue>
#include <vector>

#include "batch_tuning_table.h"
#include "batched.hpp"
#include "common.cuh"
#include "internal.hpp"
#include "plain.hpp"

namespace jsvd {
namespace {

constexpr int kLanes = 256;      // reduction width T (reference default)
constexpr int kW = kLanes / 32;  // virtual lanes per physical lane
constexpr int kClasses = 5;

// The in-warp levels 16 .. 1 of the reference's tree for the three sums of a
// pair at once: at each level a lane keeps one of two quantities and hands the
// other over (the operands of an addition commute, so each total meets in the
// reference's order).  Six exchanges instead of fifteen.  The totals end up in
// lane 0 (pp), lane 8 (pq) and lane 16 (qq); every lane returns the one of its
// lane / 8.
__device__ __forceinline__ double warp_tree3(double pp, double qq, double pq, int lane)
{
    const bool hi = (lane & 16) != 0;
    const double give = hi ? pp : qq;
    double a = hi ? qq : pp;  // pp below lane 16, qq from there
    a += __shfl_xor_sync(0xffffffffu, give, 16);
    pq += __shfl_xor_sync(0xffffffffu, pq, 16);
    const bool mid = (lane & 8) != 0;
    const double give2 = mid ? a : pq;
    double b = mid ? pq : a;
    b += __shfl_xor_sync(0xffffffffu, give2, 8);
    b += __shfl_xor_sync(0xffffffffu, b, 4);
    b += __shfl_xor_sync(0xffffffffu, b, 2);
    b += __shfl_xor_sync(0xffffffffu, b, 1);
    return b;
}

// Reference-order dot products of columns x, y (length m) by one warp, as
// warp_tree3 returns them.  NJ > 0: at most 32 NJ rows (NJ <= kW), one per
// virtual lane and none beyond; NJ = 0: any number.  A virtual lane's single
// product is its sum (fma with a zero rounds it the same way).
template <int NJ>
__device__ __forceinline__ double warp_pair_stats(const double *x, const double *y, int m, int lane)
{
    constexpr int J = NJ > 0 ? NJ : kW;
    double app[J], aqq[J], apq[J];
    if constexpr (NJ > 0) {
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int r = 32 * j + lane;
            app[j] = aqq[j] = apq[j] = 0.0;
            if (r < m) {
                const double a = x[r], b = y[r];
                app[j] = a * a;
                aqq[j] = b * b;
                apq[j] = a * b;
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < J; ++j) app[j] = aqq[j] = apq[j] = 0.0;
        for (int base = 0; base < m; base += kLanes) {
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int r = base + 32 * j + lane;
                if (r < m) {
                    const double a = x[r], b = y[r];
                    app[j] = fma(a, a, app[j]);
                    aqq[j] = fma(b, b, aqq[j]);
                    apq[j] = fma(a, b, apq[j]);
                }
            }
        }
    }
#pragma unroll
    for (int s = J / 2; s >= 1; s >>= 1)
#pragma unroll
        for (int w = 0; w < s; ++w) {
            app[w] += app[w + s];
            aqq[w] += aqq[w + s];
            apq[w] += apq[w + s];
        }
    return warp_tree3(app[0], aqq[0], apq[0], lane);
}

// Rotation of one column pair of A (length m) and of V (length n) by one
// warp.  Each 256-row chunk of all four columns is loaded into registers
// before any store: with the working copies in global memory a load -> rotate
// -> store loop pays one L2 round trip per 32 rows, because the compiler cannot
// move a load past a store to a possibly aliasing column.
// NJ > 0: m and n are at most 32 NJ; NJ = 0: any length.  kApart (everything in
// shared memory, where the round trip is short): A's columns first, then V's,
// in half the registers.
template <int J>
__device__ __forceinline__ void warp_rotate_columns(double *x, double *y, int m, int lane, double c, double s)
{
    double xa[J], ya[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int r = 32 * j + lane;
        if (r < m) {
            xa[j] = x[r];
            ya[j] = y[r];
        }
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int r = 32 * j + lane;
        if (r < m) {
            x[r] = rot_p(c, s, xa[j], ya[j]);
            y[r] = rot_q(c, s, xa[j], ya[j]);
        }
    }
}

template <int NJ, bool kApart>
__device__ __forceinline__ void warp_rotate(double *x, double *y, int m, double *vx, double *vy, int n, int lane,
                                            double c, double s)
{
    if constexpr (NJ > 0 && kApart) {
        warp_rotate_columns<NJ>(x, y, m, lane, c, s);
        warp_rotate_columns<NJ>(vx, vy, n, lane, c, s);
        return;
    }
    constexpr int J = NJ > 0 ? NJ : kW;
    const int len = NJ > 0 ? 1 : (m > n ? m : n);
    for (int base = 0; base < len; base += kLanes) {
        double xa[J], ya[J], xv[J], yv[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int r = base + 32 * j + lane;
            if (r < m) {
                xa[j] = x[r];
                ya[j] = y[r];
            }
            if (r < n) {
                xv[j] = vx[r];
                yv[j] = vy[r];
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int r = base + 32 * j + lane;
            if (r < m) {
                x[r] = rot_p(c, s, xa[j], ya[j]);
                y[r] = rot_q(c, s, xa[j], ya[j]);
            }
            if (r < n) {
                vx[r] = rot_p(c, s, xv[j], yv[j]);
                vy[r] = rot_q(c, s, xv[j], yv[j]);
            }
        }
    }
}

__device__ __forceinline__ double warp_norm2(const double *x, int m, int lane)
{
    double acc[kW];
#pragma unroll
    for (int j = 0; j < kW; ++j) acc[j] = 0.0;
    for (int base = 0; base < m; base += kLanes) {
#pragma unroll
        for (int j = 0; j < kW; ++j) {
            const int r = base + 32 * j + lane;
            if (r < m) acc[j] = fma(x[r], x[r], acc[j]);
        }
    }
    return __shfl_sync(0xffffffffu, warp_tree<kW>(acc), 0);
}

// Per-round scratch (pair statistics and angles): `half` is n/2 rounded up to
// an even count so the double2 angle array starts on a 16-byte boundary.
__host__ __device__ constexpr int round_half(int n) { return (n / 2 + 2) & ~1; }
__host__ __device__ constexpr size_t round_scratch_doubles(int n) { return (size_t)5 * round_half(n); }

// One sweep (every round of the circle) of an m x n member whose columns
// colA(c) and V live wherever the caller keeps them, by the whole CTA.  NJ as
// in warp_pair_stats, for members of at most 32 NJ rows.  With one pair of
// loops for any number of rows a 40-row member spent most of its instructions
// on rows that it does not have, and with the loops for every bound in one
// kernel the longest ones spilled; a kernel per bound, divisions out of the
// schedule and six exchanges per tree instead of fifteen: 3000 FP64 members of
// 16..64 rows 18.0 -> 5.8 ms, class 2 (397 members of up to 226 KiB) 24.6 ->
// 17.6, 100 members of 228 x 189 with V in global memory 48 -> 31 (B200).
template <int NJ, bool kApart, class ColA>
__device__ __forceinline__ void sweep_rounds(ColA colA, double *V, int m, int n, double eps, double *st_pp,
                                             double *st_qq, double *st_pq, double2 *st_cs, int &s_rot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int ne = n + (n & 1);
    const int rounds = n >= 2 ? ne - 1 : 0;
    const int npairs = n / 2;
    double *const st_mine = lane == 0 ? st_pp : (lane == 8 ? st_pq : st_qq);  // the total this lane holds
    for (int r = 0; r < rounds; ++r) {
        // phase 1: dot products, one warp per pair
        for (int k = warp; k < npairs; k += nwarps) {
            const int2 pq = round_robin_pair(n, r, k);
            const double total = warp_pair_stats<NJ>(colA(pq.x), colA(pq.y), m, lane);
            if (lane == 0 || lane == 8 || lane == 16) st_mine[k] = total;
        }
        __syncthreads();
        // phase 2: angles, one thread per pair
        for (int k = threadIdx.x; k < npairs; k += blockDim.x) {
            double c, s;
            if (rotation_params_flat(st_pp[k], st_qq[k], st_pq[k], eps, c, s)) s_rot = 1;
            st_cs[k] = make_double2(c, s);
        }
        __syncthreads();
        // phase 3: rotations, one warp per pair
        for (int k = warp; k < npairs; k += nwarps) {
            const double2 g = st_cs[k];
            if (g.x == 0.0) continue;
            const int2 pq = round_robin_pair(n, r, k);
            warp_rotate<NJ, kApart>(colA(pq.x), colA(pq.y), m, V + (size_t)pq.x * n, V + (size_t)pq.y * n, n, lane, g.x,
                                    g.y);
        }
        __syncthreads();
    }
}

// sweep_rounds for any number of rows beside those for few, with registers of its
// own: sharing theirs it lost 8 % to what the kernel had without them (a 500 x 40
// request of the serving core).
template <bool kApart, class ColA>
__device__ __noinline__ void tall_rounds(ColA colA, double *V, int m, int n, double eps, double *st_pp, double *st_qq,
                                         double *st_pq, double2 *st_cs, int &s_rot)
{
    sweep_rounds<0, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
}

// What a kernel knows about its members' rows: nothing, at most kLanes, at
// most kLanes / 2, or that they vary (the loops for every bound in one kernel,
// which costs the longest of them their registers).  At 512 threads one kernel
// spills: any rows, A and V in global memory (72 bytes stored, 56 loaded).
enum BatchRows { kRowsAny, kRows256, kRows128, kRowsVary };

__host__ __device__ constexpr BatchRows batch_rows(int m)
{
    return m <= kLanes / 2 ? kRows128 : (m <= kLanes ? kRows256 : kRowsAny);
}

// The same with the rows known as far as kRows says; true when some pair
// rotated.  s_rot must be 0 on entry and is 0 again on return.
template <BatchRows kRows, bool kApart, class ColA>
__device__ __forceinline__ bool batch_sweep(ColA colA, double *V, int m, int n, double eps, double *st_pp,
                                            double *st_qq, double *st_pq, double2 *st_cs, int &s_rot)
{
    constexpr bool kFew = kRows == kRows128 || kRows == kRowsVary;
    constexpr bool kMany = kRows == kRowsVary;
    if constexpr (kRows == kRowsAny) {
        sweep_rounds<0, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
    } else if constexpr (!kFew) {
        sweep_rounds<8, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
    } else {
        if (m <= 32) sweep_rounds<1, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
        else if (m <= 64) sweep_rounds<2, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
        else if (!kMany || m <= 128) sweep_rounds<4, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
        else if (m <= 256) sweep_rounds<kMany ? 8 : 4, kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
        else if constexpr (kMany) tall_rounds<kApart>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
    }
    const bool any = s_rot != 0;
    __syncthreads();  // every thread has read the flag before it is reset
    if (threadIdx.x == 0) s_rot = 0;
    return any;
}

// The launches of a class do not depend on each other, and each begins when the
// CTAs of the one before have begun, on the SMs that it leaves idle.  The end of
// such a launch: it is not complete before that one is, so that what follows it
// in the stream finds both done.  (One thread waits; the other CTAs give their
// SMs back.)
__device__ __forceinline__ void end_after_previous()
{
    if (blockIdx.x == 0 && threadIdx.x == 0) pdl_wait();
}

template <bool kAShared, bool kVShared, BatchRows kRows>
__global__ void __launch_bounds__(512) batch_kernel(const BatchDesc *__restrict__ descs, int count,
                                                    int *__restrict__ next, const void *__restrict__ a_all,
                                                    int a_is_f32, double eps, int max_sweeps,
                                                    double *__restrict__ sigma_all, double *__restrict__ v_all,
                                                    double *__restrict__ u_all, int *__restrict__ sweeps_all,
                                                    double *__restrict__ workspace, size_t ws_stride,
                                                    int smem_doubles)
{
    // A and V in global memory: the leading columns of A that fit the shared
    // memory left over live there instead (a pair reads its columns from
    // whichever space holds them).
    constexpr bool kHybrid = !kAShared && !kVShared;
    extern __shared__ double smem[];
    __shared__ int s_idx;
    __shared__ int s_rot;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    double *gws = workspace + (size_t)blockIdx.x * ws_stride;
    pdl_launch_dependents();
    for (;;) {
        if (threadIdx.x == 0) s_idx = atomicAdd(next, 1);
        __syncthreads();
        const int idx = s_idx;
        if (idx >= count) return end_after_previous();
        const BatchDesc d = descs[idx];
        const int m = d.m, n = d.n;
        const int half = round_half(n);
        // smem layout: [round scratch 5*half][A if shared][V if shared]
        double *st_pp = smem, *st_qq = smem + half, *st_pq = smem + 2 * half;
        double2 *st_cs = reinterpret_cast<double2 *>(smem + 3 * half);  // 2*half doubles, 16-byte aligned
        double *sm_rest = smem + round_scratch_doubles(n);
        double *A = kAShared ? sm_rest : gws;
        double *V = kVShared ? (kAShared ? sm_rest + (size_t)m * n : gws + (size_t)m * n)
                             : (kAShared ? gws : gws + (size_t)m * n);
        // columns 0 .. ks-1 of A in shared memory, ks .. n-1 in the global slice
        const int ks = kHybrid ? max(0, min(n, (smem_doubles - (int)round_scratch_doubles(n)) / m)) : 0;
        auto colA = [&](int c) -> double * {
            if constexpr (kHybrid) return c < ks ? sm_rest + (size_t)c * m : gws + (size_t)(c - ks) * m;
            else return A + (size_t)c * m;
        };
        const size_t mn = (size_t)m * n;
        if (a_is_f32) {
            const float *src = reinterpret_cast<const float *>(a_all) + d.a_off;
            for (size_t e = threadIdx.x; e < mn; e += blockDim.x) {
                const size_t r = e / n, c = e - r * n;
                colA((int)c)[r] = (double)src[e];
            }
        } else {
            const double *src = reinterpret_cast<const double *>(a_all) + d.a_off;
            for (size_t e = threadIdx.x; e < mn; e += blockDim.x) {
                const size_t r = e / n, c = e - r * n;
                colA((int)c)[r] = src[e];
            }
        }
        for (size_t e = threadIdx.x; e < (size_t)n * n; e += blockDim.x) V[e] = (e / n == e % n) ? 1.0 : 0.0;
        if (threadIdx.x == 0) s_rot = 0;
        __syncthreads();
        int sweeps = 1;
        if (n >= 2) {
            for (int sw = 0; sw < max_sweeps; ++sw) {
                const bool any = batch_sweep<kRows, kAShared && kVShared>(colA, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
                sweeps = sw + 1;
                if (!any) break;
            }
        }
        // sigma, U (optional), V (row-major)
        double *sg = sigma_all + d.s_off;
        for (int c = warp; c < n; c += nwarps) {
            const double *x = colA(c);
            const double sc = sqrt(fmax(warp_norm2(x, m, lane), 0.0));
            if (lane == 0) sg[c] = sc;
            if (u_all != nullptr) {
                double *u = u_all + d.u_off;
                for (int i = lane; i < m; i += 32) u[(size_t)i * n + c] = (sc > eps) ? (x[i] / sc) : 0.0;
            }
        }
        if (v_all != nullptr) {
            double *vo = v_all + d.v_off;
            for (size_t e = threadIdx.x; e < (size_t)n * n; e += blockDim.x) {
                const size_t r = e / n, c = e - r * n;
                vo[e] = V[c * n + r];
            }
        }
        if (sweeps_all != nullptr && threadIdx.x == 0) sweeps_all[idx] = sweeps;
        __syncthreads();  // the working copies are reused by the next matrix
    }
}

// One sweep step of the sweep-granular batch (serving core): CTA i runs one
// sweep of member i, whose state (A and V, FP64, column-major) stays in
// global memory between steps.  On its first step (in != null) a member
// starts from its row-major FP64 input with V = I, as batch_kernel does.  A
// is worked on in shared memory, and V too when kVShared (else in place in
// the state).  rotated[i] = 1 when some pair of the sweep rotated: a member
// whose sweep did not rotate has converged, exactly where batch_kernel's
// loop over sweeps stops.
template <bool kVShared>
__global__ void __launch_bounds__(256, 2) batch_step_kernel(const StepDesc *__restrict__ descs, double eps,
                                                            int *__restrict__ rotated)
{
    extern __shared__ double smem[];
    __shared__ int s_rot;
    const StepDesc d = descs[blockIdx.x];
    const int m = d.m, n = d.n;
    const int half = round_half(n);
    double *st_pp = smem, *st_qq = smem + half, *st_pq = smem + 2 * half;
    double2 *st_cs = reinterpret_cast<double2 *>(smem + 3 * half);
    double *A = smem + round_scratch_doubles(n);
    double *gA = d.a, *gV = d.v;
    double *V = kVShared ? A + (size_t)m * n : gV;
    const size_t mn = (size_t)m * n, nn = (size_t)n * n;
    if (d.in != nullptr) {
        const double *src = d.in;
        for (size_t e = threadIdx.x; e < mn; e += blockDim.x) {
            const size_t r = e / n, c = e - r * n;
            A[c * m + r] = src[e];
        }
        for (size_t e = threadIdx.x; e < nn; e += blockDim.x) V[e] = (e / n == e % n) ? 1.0 : 0.0;
    } else {
        for (size_t e = threadIdx.x; e < mn; e += blockDim.x) A[e] = gA[e];
        if (kVShared)
            for (size_t e = threadIdx.x; e < nn; e += blockDim.x) V[e] = gV[e];
    }
    if (threadIdx.x == 0) s_rot = 0;
    __syncthreads();
    bool any = false;
    if (n >= 2) any = batch_sweep<kRowsVary, kVShared>([&](int c) { return A + (size_t)c * m; }, V, m, n, eps, st_pp, st_qq, st_pq, st_cs, s_rot);
    for (size_t e = threadIdx.x; e < mn; e += blockDim.x) gA[e] = A[e];
    if (kVShared)
        for (size_t e = threadIdx.x; e < nn; e += blockDim.x) gV[e] = V[e];
    if (threadIdx.x == 0) rotated[blockIdx.x] = any ? 1 : 0;
}

// Outputs of retired members of the sweep-granular batch: sigma, V
// (row-major) and optionally U (row-major) from the state, with
// batch_kernel's formulas (CTA i: member i).
__global__ void __launch_bounds__(256) batch_finish_kernel(const StepDesc *__restrict__ descs, double eps)
{
    const StepDesc d = descs[blockIdx.x];
    const int m = d.m, n = d.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const double *gA = d.a, *gV = d.v;
    double *sg = d.s_out;
    for (int c = warp; c < n; c += nwarps) {
        const double *x = gA + (size_t)c * m;
        const double sc = sqrt(fmax(warp_norm2(x, m, lane), 0.0));
        if (lane == 0) sg[c] = sc;
        if (d.u_out != nullptr) {
            double *u = d.u_out;
            for (int i = lane; i < m; i += 32) u[(size_t)i * n + c] = (sc > eps) ? (x[i] / sc) : 0.0;
        }
    }
    double *vo = d.v_out;
    for (size_t e = threadIdx.x; e < (size_t)n * n; e += blockDim.x) {
        const size_t r = e / n, c = e - r * n;
        vo[e] = gV[c * n + r];
    }
}

// ---- cluster classes ----------------------------------------------------------
// A member whose A and V do not fit one CTA's shared memory is solved by a
// cluster of C CTAs (C = 2, 4, 8) with A and V spread over the cluster's
// distributed shared memory, laid out as the round-robin circle itself.
// CTA i owns the contiguous pair slots [k0, k1) of the circle (slot k =
// positions k and ne-1-k, the pair (top, bottom)) and one warp works a slot.
// Between rounds the top row moves one slot right and the bottom row one slot
// left (position 0 stays; ne-1 goes to 1, half-1 to half), so inside a CTA no
// column moves at all: the top slots live in a ring of S+1 column buffers
// indexed (j - g) mod (S+1) at round g, the bottom slots in a ring indexed
// (j + g) mod (S+1), and the spare buffer of each ring receives the one
// column that arrives for round g+1.  Per round a CTA sends two columns: its
// last top column to the right neighbour's spare top buffer and its first
// bottom column to the left neighbour's spare bottom buffer (both written
// straight from the rotation's registers over distributed shared memory; the
// two end CTAs send one of them to themselves).  One cluster barrier per
// round.  A buffer holds a column of A (m) followed by the same column of V
// (n), rotated together.  Pair arithmetic is batch_kernel's (warp-per-pair
// dot products in the T = 256 order, Rutishauser angle, rot_p / rot_q), so
// every member stays bit-identical to the plain path.
//
// What bounds it (B200, 228 x 189 members on 8 CTAs of 12 slots): one member
// alone takes 2.9 us per round, a chain of dot products (0.5 us), angle (0.5),
// rotation (0.8, at the shared-memory port's rate) and the cluster barrier; two
// members on the same SMs take 3.0 us for both.  So many members share SMs by
// two where their shape allows it (cluster_choice).  Registers decide
// the rest: at two CTAs per SM a thread has 80, and with the member's shape and
// the ring indices of every buffer kept in them the loops' own values went to
// local memory (5.2 us per round; in shared memory now, ClusterRound; 12 to 16
// bytes still spill, 64 stored and 96 loaded in the form for more than 256 rows,
// which cluster_choice takes the less often).  100
// members: 21.5 ms, 31.3 on one CTA each; an SM per CTA with two slots in half
// of its warps took 29.

// Threads of a cluster CTA with an SM to itself, and of one that shares it
// with a CTA of another cluster.
constexpr int kClusterThreads = 512, kClusterThreadsShared = 384;
constexpr int kClusterMaxSlots = 64;  // pair slots per CTA

__host__ __device__ constexpr int cluster_slots_max(int n, int C) { return ((n + (n & 1)) / 2 + C - 1) / C; }

// Column buffer length: A's m rows, then V's n rows, each padded to whole warps
// (the padding rows are rotated and moved like the others; A's are zero).
__host__ __device__ constexpr int cluster_rows(int m) { return (m + 31) & ~31; }
__host__ __device__ constexpr int cluster_ld(int m, int n) { return cluster_rows(m) + cluster_rows(n); }

// Shared memory of one CTA: column 0's fixed buffer and two rings.
__host__ __device__ constexpr size_t cluster_smem_bytes(int m, int n, int C)
{
    return sizeof(double) * (size_t)(2 * cluster_slots_max(n, C) + 3) * (size_t)cluster_ld(m, n);
}

__device__ __forceinline__ int pmod(int a, int b)
{
    const int r = a % b;
    return r < 0 ? r + b : r;
}

// Address of this CTA's shared-memory location `p` in the shared memory of
// CTA `rank` of the cluster (a shared::cluster address).
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank)
{
    uint32_t out;
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(rank));
    return out;
}

__device__ __forceinline__ void st_cluster(uint32_t addr, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// Moves one column (ld rows) to a shared::cluster address.
__device__ __forceinline__ void warp_move_cl(const double *x, uint32_t xo, int ld, int lane)
{
    for (int r = lane; r < ld; r += 32) st_cluster(xo + 8u * (uint32_t)r, x[r]);
}

// Rotation of a column pair in this CTA's buffers (ld rows, a multiple of 32),
// in place, four chunks loaded before any is stored.
__device__ __forceinline__ void warp_rotate_local(double *x, double *y, int ld, int lane, double c, double s)
{
    x += lane;
    y += lane;
    int r = 0;
    for (; r + 128 <= ld; r += 128) {
        double xv[4], yv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            xv[j] = x[r + 32 * j];
            yv[j] = y[r + 32 * j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            x[r + 32 * j] = rot_p(c, s, xv[j], yv[j]);
            y[r + 32 * j] = rot_q(c, s, xv[j], yv[j]);
        }
    }
    double xv[3], yv[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (r + 32 * j < ld) {
            xv[j] = x[r + 32 * j];
            yv[j] = y[r + 32 * j];
        }
#pragma unroll
    for (int j = 0; j < 3; ++j)
        if (r + 32 * j < ld) {
            x[r + 32 * j] = rot_p(c, s, xv[j], yv[j]);
            y[r + 32 * j] = rot_q(c, s, xv[j], yv[j]);
        }
}

// The same to the shared::cluster addresses xo and yo of the columns' next
// buffers.
__device__ __forceinline__ void warp_rotate_away(const double *x, const double *y, uint32_t xo, uint32_t yo, int ld,
                                                 int lane, double c, double s)
{
    x += lane;
    y += lane;
    xo += 8u * (uint32_t)lane;
    yo += 8u * (uint32_t)lane;
    int r = 0;
    for (; r + 128 <= ld; r += 128) {
        double xv[4], yv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            xv[j] = x[r + 32 * j];
            yv[j] = y[r + 32 * j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            st_cluster(xo + 8u * (uint32_t)(r + 32 * j), rot_p(c, s, xv[j], yv[j]));
            st_cluster(yo + 8u * (uint32_t)(r + 32 * j), rot_q(c, s, xv[j], yv[j]));
        }
    }
    for (; r < ld; r += 32) {
        const double xv = x[r], yv = y[r];
        st_cluster(xo + 8u * (uint32_t)r, rot_p(c, s, xv, yv));
        st_cluster(yo + 8u * (uint32_t)r, rot_q(c, s, xv, yv));
    }
}

// Angle of a slot's pair of columns (mp rows of A in whole chunks, padded with
// zeros; m real ones); false when it does not rotate.  kTall: more than kLanes
// rows.
template <bool kTall>
__device__ __forceinline__ bool warp_angle_cl(const double *x, const double *y, int m, int mp, int lane, double eps,
                                              double &c, double &s)
{
    double total;
    if constexpr (kTall) {
        total = warp_pair_stats<0>(x, y, m, lane);
    } else {
        double xr[kW], yr[kW];
#pragma unroll
        for (int j = 0; j < kW; ++j) {
            const bool in = 32 * j < mp;
            xr[j] = in ? x[32 * j + lane] : 0.0;
            yr[j] = in ? y[32 * j + lane] : 0.0;
        }
        // the register levels of the tree, s[j] += s[j + 4], + 2, + 1, one sum
        // after the other
        auto sum = [](const double(&a)[kW], const double(&b)[kW]) {
            return ((a[0] * b[0] + a[4] * b[4]) + (a[2] * b[2] + a[6] * b[6])) +
                   ((a[1] * b[1] + a[5] * b[5]) + (a[3] * b[3] + a[7] * b[7]));
        };
        total = warp_tree3(sum(xr, xr), sum(yr, yr), sum(xr, yr), lane);
    }
    const double pp = __shfl_sync(0xffffffffu, total, 0);
    const double pq = __shfl_sync(0xffffffffu, total, 8);
    const double qq = __shfl_sync(0xffffffffu, total, 16);
    // Far below the threshold (by a factor of two, well above the rounding of
    // either side) nothing rotates: most pairs of the last sweeps stop here.
    if (pq * pq < (0.25 * eps * eps) * (fmax(pp, 0.0) * fmax(qq, 0.0))) return false;
    return rotation_params_flat(pp, qq, pq, eps, c, s);
}

// A CTA's share of a member: its slots [k0, k0 + S) of the circle's half, and
// its buffers (offsets in doubles): column 0's fixed one (CTA 0 only, where slot
// 0's top never moves: jt0 = 1), the top ring of rt buffers and the bottom ring
// of rb.  Top slot j is in top buffer (j - jt0 - g) mod rt at round g, bottom
// slot j in bottom buffer (j + g) mod rb.
struct ClusterShare {
    int m, n, ne, half, L, ld, mp, k0, S, jt0, rt, rb, top_off, bot_off;
    __device__ ClusterShare(int m_, int n_, int rank, int C) : m(m_), n(n_)
    {
        ne = n + (n & 1);
        half = ne / 2;
        L = ne - 1;
        ld = cluster_ld(m, n);
        mp = cluster_rows(m);
        k0 = rank * half / C;
        S = (rank + 1) * half / C - k0;  // >= 2 (host: half >= 2C)
        jt0 = rank == 0 ? 1 : 0;
        rt = S - jt0 + 1;
        rb = S + 1;
        top_off = ld;
        bot_off = (cluster_slots_max(n, C) + 2) * ld;
    }
    __device__ int top_at(int j, int g) const { return jt0 && j == 0 ? 0 : top_off + pmod(j - jt0 - g, rt) * ld; }
    __device__ int bot_at(int j, int g) const { return bot_off + pmod(j + g, rb) * ld; }
};

// What a round needs besides: g modulo the rings' lengths, the slot of this CTA
// that holds the dummy column of an odd n (or -1) and in which position, and
// the shared::cluster addresses that the last slot's top column and the first
// slot's bottom column move to.  One thread works it out a round ahead, in
// shared memory: kept in every thread's registers, this and the member's shape
// pushed the loops' own values into local memory.
struct ClusterRound {
    int gt, gb, dummy, dummy_top;
    uint32_t top_to, bot_to;
};
struct ClusterKeep {
    int idx, m, n;     // the member
    int dpos;          // circle position of the dummy column
    int o_top, o_bot;  // ring buffers that receive this CTA's outgoing columns
    int s_right, s_left;
};

__device__ __forceinline__ void cluster_round(const ClusterShare &sh, int rank, int C, const ClusterKeep &kp,
                                              uint32_t self, uint32_t right, uint32_t left, int gt, int gb,
                                              ClusterRound &out)
{
    out.gt = gt;
    out.gb = gb;
    out.dummy_top = kp.dpos < sh.half;
    const int d = (out.dummy_top ? kp.dpos : sh.L - kp.dpos) - sh.k0;
    out.dummy = (sh.n & 1) && d >= 0 && d < sh.S ? d : -1;
    out.top_to = rank < C - 1 ? right + 8u * (uint32_t)(sh.top_off + kp.o_top * sh.ld)
                              : self + 8u * (uint32_t)(sh.bot_off + kp.o_top * sh.ld);
    out.bot_to = rank > 0 ? left + 8u * (uint32_t)(sh.bot_off + kp.o_bot * sh.ld)
                          : self + 8u * (uint32_t)(sh.top_off + kp.o_bot * sh.ld);
}

// A member's descriptor, read anew each time (not kept in registers).
__device__ __forceinline__ BatchDesc read_desc(const BatchDesc *descs, int idx)
{
    const volatile BatchDesc *p = descs + idx;
    BatchDesc d;
    d.m = p->m;
    d.n = p->n;
    d.a_off = p->a_off;
    d.s_off = p->s_off;
    d.v_off = p->v_off;
    d.u_off = p->u_off;
    return d;
}

template <int C, bool kTall, bool kShare>
__global__ void __launch_bounds__(kShare ? kClusterThreadsShared : kClusterThreads, kShare ? 2 : 1)
    batch_cluster_kernel(const BatchDesc *__restrict__ descs, int count, int *__restrict__ next,
                         const void *__restrict__ a_all, int a_is_f32, double eps, int max_sweeps,
                         double *__restrict__ sigma_all, double *__restrict__ v_all, double *__restrict__ u_all,
                         int *__restrict__ sweeps_all)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) double smem[];
    __shared__ int s_idx;
    __shared__ int s_rot;
    __shared__ unsigned long long s_stamp;  // rank 0's copy: last (member, sweep) stamp that rotated
    __shared__ ClusterKeep s_keep;
    __shared__ __align__(16) ClusterRound s_round[2];  // by round parity
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int nwarps = (kShare ? kClusterThreadsShared : kClusterThreads) / 32;
    constexpr int kKeeper = 64;  // the thread that looks a round ahead
    if (threadIdx.x == 0) {
        s_rot = 0;
        s_stamp = 0;
    }
    pdl_launch_dependents();
    for (;;) {
        int ld, mp, m, rounds, S, jt0, bot_base;
        {
            const int rank = (int)cluster.block_rank();
            if (rank == 0 && threadIdx.x == 0) s_idx = atomicAdd(next, 1);
            cluster.sync();  // (the first one also orders the initialisation above)
            const int idx = *(volatile const int *)cluster.map_shared_rank(&s_idx, 0);
            // every CTA has read the index and finished the previous member's
            // outputs before any CTA writes into another's buffers or exits
            cluster.sync();
            if (idx >= count) return end_after_previous();
            const BatchDesc d = read_desc(descs, idx);
            const ClusterShare sh(d.m, d.n, rank, C);
            // round 0: position p holds column p; V = I
            const int ncl = 2 * sh.S;
            for (int e = threadIdx.x; e < sh.mp * ncl; e += blockDim.x) {
                const int row = e / ncl, cc = e - row * ncl;
                const int j = cc < sh.S ? cc : cc - sh.S;
                const int col = cc < sh.S ? sh.k0 + j : sh.ne - 1 - (sh.k0 + j);
                if (col >= sh.n) continue;  // the dummy column of an odd n
                const size_t src = (size_t)d.a_off + (size_t)row * sh.n + col;
                smem[(cc < sh.S ? sh.top_at(j, 0) : sh.bot_at(j, 0)) + row] =
                    row >= sh.m ? 0.0
                                : (a_is_f32 ? (double)reinterpret_cast<const float *>(a_all)[src]
                                            : reinterpret_cast<const double *>(a_all)[src]);
            }
            for (int e = threadIdx.x; e < (sh.ld - sh.mp) * ncl; e += blockDim.x) {
                const int row = e / ncl, cc = e - row * ncl;
                const int j = cc < sh.S ? cc : cc - sh.S;
                const int col = cc < sh.S ? sh.k0 + j : sh.ne - 1 - (sh.k0 + j);
                if (col >= sh.n) continue;
                smem[(cc < sh.S ? sh.top_at(j, 0) : sh.bot_at(j, 0)) + sh.mp + row] = row == col ? 1.0 : 0.0;
            }
            if (threadIdx.x == kKeeper) {
                // the right neighbour's spare top buffer (the last CTA: its own
                // spare bottom one) and the left neighbour's spare bottom buffer
                // (CTA 0: its own spare top one)
                s_keep.idx = idx;
                s_keep.m = d.m;
                s_keep.n = d.n;
                s_keep.dpos = sh.L;
                s_keep.s_right = rank < C - 1 ? (rank + 2) * sh.half / C - (rank + 1) * sh.half / C : 0;
                s_keep.s_left = rank > 0 ? sh.k0 - (rank - 1) * sh.half / C : 0;
                s_keep.o_top = rank < C - 1 ? s_keep.s_right : sh.S;
                s_keep.o_bot = rank > 0 ? s_keep.s_left : sh.rt - 1;
                cluster_round(sh, rank, C, s_keep, cluster_addr(smem, rank),
                              cluster_addr(smem, rank < C - 1 ? rank + 1 : rank),
                              cluster_addr(smem, rank > 0 ? rank - 1 : rank), 0, 0, s_round[0]);
            }
            ld = sh.ld;
            mp = sh.mp;
            m = sh.m;
            S = sh.S;
            jt0 = sh.jt0;
            bot_base = sh.bot_off;
            rounds = sh.n >= 2 ? sh.L : 0;
        }
        __syncthreads();
        int g = 0, sweeps = 1;
        if (rounds > 0) {
            for (int sw = 0; sw < max_sweeps; ++sw) {
                for (int r = 0; r < rounds; ++r, ++g) {
                    const volatile ClusterRound &rd = s_round[g & 1];
#pragma unroll 1
                    for (int j = warp; j < S; j += nwarps) {
                        int tb = j - jt0 - rd.gt, bb = j + rd.gb;
                        if (tb < 0) tb += S - jt0 + 1;
                        if (bb > S) bb -= S + 1;
                        double *xt = smem + (jt0 && j == 0 ? 0 : (1 + tb) * ld);
                        double *xb = smem + bot_base + bb * ld;
                        const bool dummy = j == rd.dummy;
                        double c, s;
                        const bool rotates = !dummy && warp_angle_cl<kTall>(xt, xb, m, mp, lane, eps, c, s);
                        if (rotates && lane == 0) s_rot = 1;
                        if (j != 0 && j != S - 1) {
                            if (rotates) warp_rotate_local(xt, xb, ld, lane, c, s);
                            continue;
                        }
                        // a slot at the end of the CTA's row: its outer column
                        // leaves (at either end of the circle into the other
                        // ring), rotated or (the dummy's slot too) as it is
                        const uint32_t sm_self = cluster_addr(smem, (int)cluster.block_rank());
                        const uint32_t dt =
                            j == S - 1 ? rd.top_to : sm_self + (uint32_t)((const char *)xt - (const char *)smem);
                        const uint32_t db = j == 0 ? rd.bot_to : sm_self + (uint32_t)((const char *)xb - (const char *)smem);
                        if (rotates) {
                            warp_rotate_away(xt, xb, dt, db, ld, lane, c, s);
                        } else {
                            if (j == S - 1 && !(dummy && rd.dummy_top)) warp_move_cl(xt, dt, ld, lane);
                            if (j == 0 && !(dummy && !rd.dummy_top)) warp_move_cl(xb, db, ld, lane);
                        }
                    }
                    if (threadIdx.x == kKeeper) {
                        const int rank = (int)cluster.block_rank();
                        ClusterKeep kp = s_keep;
                        const ClusterShare sh(kp.m, kp.n, rank, C);
                        kp.dpos = kp.dpos == sh.L ? 1 : kp.dpos + 1;
                        if (rank < C - 1) kp.o_top = kp.o_top == 0 ? kp.s_right : kp.o_top - 1;
                        else kp.o_top = kp.o_top == sh.rb - 1 ? 0 : kp.o_top + 1;
                        if (rank > 0) kp.o_bot = kp.o_bot == kp.s_left ? 0 : kp.o_bot + 1;
                        else kp.o_bot = kp.o_bot == 0 ? sh.rt - 1 : kp.o_bot - 1;
                        s_keep = kp;
                        cluster_round(sh, rank, C, kp, cluster_addr(smem, rank),
                                      cluster_addr(smem, rank < C - 1 ? rank + 1 : rank),
                                      cluster_addr(smem, rank > 0 ? rank - 1 : rank),
                                      rd.gt == sh.rt - 1 ? 0 : rd.gt + 1, rd.gb == sh.rb - 1 ? 0 : rd.gb + 1,
                                      s_round[(g + 1) & 1]);
                    }
                    cluster.sync();
                }
                // sweep test over the cluster: a CTA that rotated raises rank 0's stamp
                unsigned long long *stamp0 = cluster.map_shared_rank(&s_stamp, 0);
                const unsigned long long stamp =
                    (unsigned long long)*(volatile int *)&s_keep.idx * (unsigned)(max_sweeps + 1) + sw + 1;
                if (threadIdx.x == 0) {
                    if (s_rot) atomicMax(stamp0, stamp);
                    s_rot = 0;
                }
                cluster.sync();
                const bool any = *(volatile const unsigned long long *)stamp0 == stamp;
                sweeps = sw + 1;
                if (!any) break;
            }
        }
        // every sweep is a whole turn of the circle: position p holds column p again
        const int rank = (int)cluster.block_rank();
        const int idx = *(volatile int *)&s_keep.idx;
        const BatchDesc d = read_desc(descs, idx);
        const ClusterShare sh(d.m, d.n, rank, C);
        double *sg = sigma_all + d.s_off;
        for (int cc = warp; cc < 2 * sh.S; cc += nwarps) {
            const int j = cc < sh.S ? cc : cc - sh.S;
            const int col = cc < sh.S ? sh.k0 + j : sh.ne - 1 - (sh.k0 + j);
            if (col >= sh.n) continue;
            const double *x = smem + (cc < sh.S ? sh.top_at(j, g) : sh.bot_at(j, g));
            const double sc = sqrt(fmax(warp_norm2(x, sh.m, lane), 0.0));
            if (lane == 0) sg[col] = sc;
            if (u_all != nullptr) {
                double *u = u_all + d.u_off;
                for (int i = lane; i < sh.m; i += 32) u[(size_t)i * sh.n + col] = (sc > eps) ? (x[i] / sc) : 0.0;
            }
            if (v_all != nullptr) {
                double *vo = v_all + d.v_off;
                for (int i = lane; i < sh.n; i += 32) vo[(size_t)i * sh.n + col] = x[sh.mp + i];
            }
        }
        if (rank == 0 && threadIdx.x == 0 && sweeps_all != nullptr) sweeps_all[idx] = sweeps;
    }
}

using ClusterFn = void (*)(const BatchDesc *, int, int *, const void *, int, double, int, double *, double *, double *,
                           int *);

template <bool kTall, bool kShare>
ClusterFn cluster_fn_c(int C)
{
    return C == 2 ? batch_cluster_kernel<2, kTall, kShare>
                  : (C == 4 ? batch_cluster_kernel<4, kTall, kShare> : batch_cluster_kernel<8, kTall, kShare>);
}

// `tall`: members of more than kLanes rows; `share`: two CTAs per SM.
ClusterFn cluster_fn(int C, bool tall, bool share)
{
    if (tall) return share ? cluster_fn_c<true, true>(C) : cluster_fn_c<true, false>(C);
    return share ? cluster_fn_c<false, true>(C) : cluster_fn_c<false, false>(C);
}

// Size classes whose members may go to clusters (bit c = class c; classes 2-4
// only; class 3 while its members are few: cluster_choice), initially the
// compiled-in tuning table's choice.  Process-wide.
#ifndef JSVD_BATCH_CLUSTER_CLASSES
#define JSVD_BATCH_CLUSTER_CLASSES (1 << 3 | 1 << 4)
#endif
std::atomic<int> g_cluster_mask{JSVD_BATCH_CLUSTER_CLASSES};  // the tuning table's choice
int batch_cluster_mask() { return g_cluster_mask.load(std::memory_order_relaxed); }

// Cluster of a member; C = 0: the class's one-CTA kernel.  share: two CTAs to an
// SM, so that one member's loads and stores run beside the other's arithmetic.
struct ClusterChoice {
    int C = 0;
    bool share = false;
};

// Work of one member per sweep, ~ n^2 (m + n): the queue order inside a class.
double member_work(int m, int n) { return (double)n * n * (m + n); }

// Clusters that the device holds at once: own[i] of 2 << i CTAs with an SM each,
// shared4 of four CTAs at two to an SM.
struct ClusterCapacity {
    int sms = 0, own[3] = {}, shared4 = 0;
};

// The cluster of an m x n member of class `cls` that has `members` in the batch.
// The larger the cluster, the sooner its member is done and the fewer run side by
// side, so the choice goes by how many have to.  ms for 14, 32, 70 and 592 equal
// members (B200):
//                        500 x 80 (class 4)   250 x 140 (class 4)   350 x 70 (class 3)
//   8 CTAs, an SM each   1.5  4.4  7.3  58    2.7  7.9   13  104    1.2  3.5  5.8  46
//   8 CTAs, shared       1.8  2.2  6.3  38    2.7  3.5  9.7   62    1.4  1.6  4.6  28
//   4 CTAs, an SM each   1.8  1.8  5.1  30    4.7  4.7   14   83    1.4  1.4  4.0  23
//   4 CTAs, shared       2.1  2.1  2.8  23    does not fit          1.6  1.6  2.5  16
//   2 CTAs, an SM each   3.1  3.1  3.1  24    does not fit          2.5  2.5  2.5  19
//   the class's kernel   7.7  7.7  7.7  31     13   13   14   54    4.1  4.1  4.1  16
// While all are resident at once: the largest cluster with an SM per CTA, before
// that eight shared CTAs where they keep the warps busy (9 to 12 slots on 12
// warps).  More members: in class 4 two CTAs where they hold the member, four
// shared ones where those keep the warps busy, else eight shared ones or the
// smallest that holds it.  In class 3 the smallest, or the class's kernel, as
// clusters_sooner decides for the class.
ClusterChoice cluster_choice(int m, int n, int cls, long members, bool sooner, size_t smem_cap,
                             const ClusterCapacity &cap)
{
    const int half = (n + (n & 1)) / 2;
    auto own = [&](int C) {  // at least two slots per CTA
        return half >= 2 * C && cluster_slots_max(n, C) <= kClusterMaxSlots && cluster_smem_bytes(m, n, C) <= smem_cap;
    };
    auto shared = [&](int C, int least) {
        const int slots = cluster_slots_max(n, C);
        return half >= 2 * C && slots >= least && slots <= kClusterThreadsShared / 32 &&
               cluster_smem_bytes(m, n, C) <= smem_cap / 2 - 1024;
    };
    if (own(8) && members <= cap.own[2]) return {8, false};
    if (shared(8, 9) && 8 * members <= 2 * cap.sms) return {8, true};
    if (own(4) && members <= cap.own[1]) return {4, false};
    const int C = own(2) ? 2 : (own(4) ? 4 : (own(8) ? 8 : 0));
    if (cls == 3) return sooner ? ClusterChoice{C, false} : ClusterChoice{};
    if (C == 2) {
        if (shared(4, 9) && (members <= cap.shared4 || members > cap.own[0])) return {4, true};
        return {2, false};
    }
    // (8 slots: 512 x 128 7.3 ms against 8.0 for 37 members, 76 against 72 for 592)
    if (shared(8, 2 * members <= cap.sms ? 8 : 9)) return {8, true};
    return {C, false};
}

// Last end of jobs of the given lengths on `at_once` workers, each job taken by
// the first free one, as the work queue does.
double makespan(const std::vector<double> &lengths, int at_once)
{
    std::priority_queue<double, std::vector<double>, std::greater<double>> ends;
    double last = 0.0;
    for (double t : lengths) {
        if ((int)ends.size() == std::max(at_once, 1)) {
            t += ends.top();
            ends.pop();
        }
        ends.push(t);
        last = std::max(last, t);
    }
    return last;
}

// Whether the smallest clusters that hold them solve the members of class 3 (in
// queue order, by work) sooner than the class's kernel does.  A member takes 1.5
// to 1.6 times as long on that kernel as on two CTAs, 1.7 to 2.2 times with more
// than 256 rows, 2.4 times as long as on four (B200); the device holds twice or
// four times as many of them.  So few members, and equal ones that fill the
// kernel's last wave badly, go to clusters (300 of 270 x 100: 18.2 ms, 23.9 on
// the class's kernel), ragged ones in number do not (211 of 100 to 226 KiB: 25.3
// ms, 45).
bool clusters_sooner(const std::vector<int> &members, const std::vector<BatchDesc> &all, size_t smem_cap,
                     const ClusterCapacity &cap)
{
    if (members.size() > 8 * (size_t)cap.sms) return false;
    std::vector<double> single, cluster[3];
    for (int i : members) {
        const int m = all[i].m, n = all[i].n;
        const double t = member_work(m, n);
        single.push_back(t);
        int c = 0;
        while (c < 3 && cluster_smem_bytes(m, n, 2 << c) > smem_cap) ++c;
        if (c == 3) return false;
        cluster[c].push_back(t / (c == 0 ? (m > kLanes ? 1.8 : 1.5) : (c == 1 ? 2.4 : 4.0)));
    }
    double ends = 0.0;
    for (int c = 0; c < 3; ++c) ends += makespan(cluster[c], cap.own[c]);
    return ends < 0.97 * makespan(single, cap.sms);
}

int cluster_capacity(int dev, int sms, size_t smem_cap, ClusterCapacity &cap)
{
    static std::atomic<int> known[64][4];
    cap.sms = sms;
    for (int i = 0; i < 4; ++i) {
        int &out = i < 3 ? cap.own[i] : cap.shared4;
        out = dev >= 0 && dev < 64 ? known[dev][i].load(std::memory_order_relaxed) : 0;
        if (out > 0) continue;
        const int C = i < 3 ? 2 << i : 4;
        const ClusterFn fn = cluster_fn(C, false, i == 3);
        JSVD_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cap));
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)C;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)C);
        lc.blockDim = dim3(i == 3 ? kClusterThreadsShared : kClusterThreads);
        lc.dynamicSmemBytes = i == 3 ? smem_cap / 2 - 1024 : smem_cap;
        lc.attrs = at;
        lc.numAttrs = 1;
        JSVD_CUDA_TRY(cudaOccupancyMaxActiveClusters(&out, fn, &lc));
        if (dev >= 0 && dev < 64) known[dev][i].store(out, std::memory_order_relaxed);
    }
    return JSVD_OK;
}

using BatchFn = void (*)(const BatchDesc *, int, int *, const void *, int, double, int, double *, double *,
                         double *, int *, double *, size_t, int);

// The one-CTA kernel of a class and of members whose rows are known as far as
// `rows` says.
BatchFn batch_fn(int cls, BatchRows rows)
{
    if (cls <= 2)
        return rows == kRows128 ? batch_kernel<true, true, kRows128>
                                : (rows == kRows256 ? batch_kernel<true, true, kRows256> : batch_kernel<true, true, kRowsAny>);
    if (cls == 3) return rows == kRowsAny ? batch_kernel<true, false, kRowsAny> : batch_kernel<true, false, kRows256>;
    return rows == kRowsAny ? batch_kernel<false, false, kRowsAny> : batch_kernel<false, false, kRows256>;
}

// Per-thread timing events: whole call and one pair per size class.
struct ThreadEvents {
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    cudaEvent_t c0[kClasses] = {}, c1[kClasses] = {};
    int device = -1;
    ~ThreadEvents()
    {
        for (int c = 0; c < kClasses; ++c) {
            if (c0[c]) cudaEventDestroy(c0[c]);
            if (c1[c]) cudaEventDestroy(c1[c]);
        }
        if (t0) cudaEventDestroy(t0);
        if (t1) cudaEventDestroy(t1);
    }
};

int thread_events(int dev, ThreadEvents **out)
{
    thread_local ThreadEvents ts;
    if (ts.device != dev) {
        if (ts.device >= 0) return invalid_argument("The batched solver is bound to the first device it ran on.");
        for (int c = 0; c < kClasses; ++c) {
            JSVD_CUDA_TRY(cudaEventCreate(&ts.c0[c]));
            JSVD_CUDA_TRY(cudaEventCreate(&ts.c1[c]));
        }
        JSVD_CUDA_TRY(cudaEventCreate(&ts.t0));
        JSVD_CUDA_TRY(cudaEventCreate(&ts.t1));
        ts.device = dev;
    }
    *out = &ts;
    return JSVD_OK;
}

constexpr jsvd_batch_tuning kBuiltinTuning[kClasses] = JSVD_BATCH_TUNING_TABLE;

// Where each class keeps its working copies (see the file comment).
constexpr bool class_a_shared(int c) { return c <= 3; }
constexpr bool class_v_shared(int c) { return c <= 2; }

// Largest dynamic shared memory a batch CTA asks for: the opt-in limit less
// 1 KiB for the static variables.
int batch_smem_cap(int dev, size_t *cap)
{
    int smem_optin = 0;
    JSVD_CUDA_TRY(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    *cap = (size_t)std::min(smem_optin, 227 * 1024) - 1024;
    return JSVD_OK;
}

// Size class of an m x n member and the shared-memory bytes it needs there.
int member_class(int m, int n, size_t smem_cap, size_t *smem_need)
{
    const size_t scratch = sizeof(double) * round_scratch_doubles(n);
    const size_t a_bytes = sizeof(double) * (size_t)m * n, v_bytes = sizeof(double) * (size_t)n * n;
    int c;
    if (scratch + a_bytes + v_bytes <= 48 * 1024) c = 0;
    else if (scratch + a_bytes + v_bytes <= 100 * 1024) c = 1;
    else if (scratch + a_bytes + v_bytes <= smem_cap) c = 2;
    else if (scratch + a_bytes <= smem_cap) c = 3;
    else c = 4;
    if (smem_need)
        *smem_need = scratch + (class_a_shared(c) ? a_bytes : 0) + (class_v_shared(c) ? v_bytes : 0);
    return c;
}

// Argument checks shared by the solver and the autotuner.
int check_batch_args(int count, const int *rows, const int *cols, const long long *a_offsets, const void *d_a,
                     bool sigma_missing, const jsvd_config &c)
{
    if (count < 0) return invalid_argument("count must be non-negative.");
    if (count > 0 && (rows == nullptr || cols == nullptr || a_offsets == nullptr || d_a == nullptr || sigma_missing))
        return invalid_argument("Batch buffers must not be null.");
    if (!(c.epsilon > 0.0)) return invalid_argument("epsilon must be positive.");
    if (c.max_sweeps <= 0) return invalid_argument("max_sweeps must be positive.");
    if (reduction_lanes(c.threads_per_block) != 256)
        return invalid_argument("The batched solver reduces with threads_per_block = 256.");
    return JSVD_OK;
}

}  // namespace

BatchStats &batch_stats()
{
    thread_local BatchStats s;
    return s;
}

int batch_solve(const BatchRequest &req, cudaStream_t stream)
{
    const int count = req.count;
    if (count <= 0) return JSVD_OK;
    int dev = 0;
    JSVD_CUDA_TRY(cudaGetDevice(&dev));
    int sms = 0;
    JSVD_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    size_t smem_cap = 0;
    int rc = batch_smem_cap(dev, &smem_cap);
    if (rc != JSVD_OK) return rc;
    ThreadEvents *ts = nullptr;
    rc = thread_events(dev, &ts);
    if (rc != JSVD_OK) return rc;

    struct Class {
        int threads;
        int ctas_per_sm;
        bool a_shared, v_shared;
    };
    Class classes[kClasses];
    int max_ctas[kClasses] = {};
    for (int c = 0; c < kClasses; ++c) {
        classes[c].threads = kBuiltinTuning[c].threads;
        classes[c].ctas_per_sm = kBuiltinTuning[c].ctas_per_sm;
        classes[c].a_shared = class_a_shared(c);
        classes[c].v_shared = class_v_shared(c);
        max_ctas[c] = kBuiltinTuning[c].max_ctas;
    }
    if (req.tuning != nullptr) {
        for (int c = 0; c < kClasses; ++c) {
            const jsvd_batch_tuning &t = req.tuning[c];
            if (t.threads < 0 || t.threads > 512 || t.threads % 32 != 0 || t.ctas_per_sm < 0 || t.max_ctas < 0)
                return invalid_argument("Batch tuning: threads must be a multiple of 32 up to 512, counts >= 0.");
            if (t.threads > 0) classes[c].threads = t.threads;
            if (t.ctas_per_sm > 0) classes[c].ctas_per_sm = t.ctas_per_sm;
            if (t.threads > 0 || t.ctas_per_sm > 0 || t.max_ctas > 0) max_ctas[c] = t.max_ctas;
        }
    }
    std::vector<std::vector<int>> members(kClasses);
    std::vector<BatchDesc> all(count);
    std::vector<size_t> need_smem(count);
    size_t s_off = 0, v_off = 0, u_off = 0;
    for (int i = 0; i < count; ++i) {
        BatchDesc d;
        d.m = req.rows[i];
        d.n = req.cols[i];
        if (d.m <= 0 || d.n <= 0 || d.m < d.n)
            return invalid_argument("Batch matrix shape must satisfy rows >= columns > 0.");
        if (dims_out_of_range((size_t)d.m, (size_t)d.n)) {
            set_last_error(JSVD_ERR_OVERFLOW, "Matrix dimensions exceed the supported range.");
            return JSVD_ERR_OVERFLOW;
        }
        d.a_off = req.a_offsets[i];
        d.s_off = (long long)s_off;
        d.v_off = (long long)v_off;
        d.u_off = (long long)u_off;
        s_off += d.n;
        v_off += (size_t)d.n * d.n;
        u_off += (size_t)d.m * d.n;
        all[i] = d;
        members[member_class(d.m, d.n, smem_cap, &need_smem[i])].push_back(i);
    }
    // Launch groups in launch order: per class, largest first, the members
    // solved by clusters of 8, 4 and 2 CTAs (classes whose bit is set in the
    // cluster mask), then the rest by the class's own kernel.  Largest work
    // first inside each group (tail balance of the work queue).
    struct Group {
        int cls, csize;
        bool tall, share;
        BatchRows rows;
        int first, count;
        size_t smem, gws;
        int grid, threads;
    };
    auto work = [&](int i) { return member_work(all[i].m, all[i].n); };
    const int mask = batch_cluster_mask();
    ClusterCapacity capacity;
    if (mask != 0)
        if (const int rc = cluster_capacity(dev, sms, smem_cap, capacity); rc != JSVD_OK) return rc;
    std::vector<Group> groups;
    std::vector<BatchDesc> ordered;
    ordered.reserve(count);
    std::vector<int> order_index;
    order_index.reserve(count);
    for (int c = kClasses - 1; c >= 0; --c) {
        std::sort(members[c].begin(), members[c].end(), [&](int x, int y) { return work(x) > work(y); });
        // by kernel: own (0-2, by rows), clusters of 2, 4, 8 (3-5), + 3 sharing an
        // SM, + 6 tall
        std::vector<int> sub[15];
        // (a launch shape given for class 3 is its own kernel's)
        const bool on = (mask >> c) & 1 && !(c == 3 && req.tuning != nullptr && req.tuning[3].threads > 0);
        const bool sooner = on && c == 3 && clusters_sooner(members[c], all, smem_cap, capacity);
        for (int i : members[c]) {
            ClusterChoice cc;
            if (on) cc = cluster_choice(all[i].m, all[i].n, c, (long)members[c].size(), sooner, smem_cap, capacity);
            const BatchRows rows = c <= 2 ? batch_rows(all[i].m) : std::min(batch_rows(all[i].m), kRows256);
            sub[cc.C == 0 ? (int)rows
                          : (cc.C == 2 ? 3 : (cc.C == 4 ? 4 : 5)) + (cc.share ? 3 : 0) + (all[i].m > kLanes ? 6 : 0)]
                .push_back(i);
        }
        for (int s : {14, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 0, 1, 2}) {
            if (sub[s].empty()) continue;
            const int k = s < 3 ? 0 : s - 3;
            Group g{c, s < 3 ? 0 : (1 << (k % 3 + 1)), s >= 3 && k >= 6, s >= 3 && k / 3 % 2 == 1, (BatchRows)std::min(s, 2),
                    (int)ordered.size(), (int)sub[s].size(), 0, 0, 0, 0};
            for (int i : sub[s]) {
                ordered.push_back(all[i]);
                order_index.push_back(i);
                if (g.csize > 0) {
                    g.smem = std::max(g.smem, cluster_smem_bytes(all[i].m, all[i].n, g.csize));
                } else {
                    g.smem = std::max(g.smem, need_smem[i]);
                    size_t w = 0;
                    if (!classes[c].a_shared) w += (size_t)all[i].m * all[i].n;
                    if (!classes[c].v_shared) w += (size_t)all[i].n * all[i].n;
                    g.gws = std::max(g.gws, w);
                }
            }
            groups.push_back(g);
        }
    }
    std::vector<size_t> gws_base(groups.size(), 0);
    size_t gws_total = 0;
    for (size_t k = 0; k < groups.size(); ++k) {
        Group &g = groups[k];
        if (g.csize > 0) {
            JSVD_CUDA_TRY(cudaFuncSetAttribute(cluster_fn(g.csize, g.tall, g.share), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem_cap));
            cudaLaunchConfig_t lc = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = (unsigned)g.csize;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            lc.gridDim = dim3((unsigned)g.csize);
            lc.blockDim = dim3(g.share ? kClusterThreadsShared : kClusterThreads);
            lc.dynamicSmemBytes = g.smem;
            lc.attrs = at;
            lc.numAttrs = 1;
            int clusters = 0;
            JSVD_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, cluster_fn(g.csize, g.tall, g.share), &lc));
            if (clusters <= 0) {
                set_last_error(JSVD_ERR_RUNTIME, "No cluster of the batched solver fits the device.");
                return JSVD_ERR_RUNTIME;
            }
            g.grid = std::min(g.count, clusters) * g.csize;
        } else {
            const Class &cl = classes[g.cls];
            g.threads = cl.threads;
            int ctas_per_sm = cl.ctas_per_sm;
            // The table's shapes suit many members per resident CTA.  Up to one
            // and a half, the last ones decide: half as many CTAs of twice the
            // warps (740 members of class 0: 4.5 -> 3.1 ms, 365 of class 1: 8.4
            // -> 6.2; at five per CTA and more the table's are the faster, 4.1
            // -> 3.3 ms for 2921 members), and a CTA to itself for every member
            // when the SMs suffice (79 of class 1: 2.2 -> 1.8 ms).
            if (req.tuning == nullptr && 2 * g.count <= 3 * sms * ctas_per_sm && ctas_per_sm > 1) {
                const int share = g.count <= sms ? ctas_per_sm : 2;
                g.threads = std::min(512, g.threads * share);
                ctas_per_sm = std::max(1, ctas_per_sm / share);
            }
            g.grid = std::min(g.count, sms * ctas_per_sm);
            if (max_ctas[g.cls] > 0) g.grid = std::min(g.grid, max_ctas[g.cls]);
            gws_base[k] = gws_total;
            gws_total += g.gws * (size_t)g.grid;
        }
    }

    BatchDesc *d_desc = nullptr;
    int *d_next = nullptr, *d_sweeps = nullptr;
    double *d_ws = nullptr;
    ScopeExit free_buffers([&] {  // stream-ordered, on every return path
        if (d_desc) cudaFreeAsync(d_desc, stream);
        if (d_next) cudaFreeAsync(d_next, stream);
        if (d_sweeps) cudaFreeAsync(d_sweeps, stream);
        if (d_ws) cudaFreeAsync(d_ws, stream);
    });
    const size_t ngroups = std::max<size_t>(groups.size(), 1);
    JSVD_CUDA_TRY(cudaMallocAsync(&d_desc, sizeof(BatchDesc) * ordered.size(), stream));
    JSVD_CUDA_TRY(cudaMallocAsync(&d_next, sizeof(int) * ngroups, stream));
    JSVD_CUDA_TRY(cudaMallocAsync(&d_sweeps, sizeof(int) * (size_t)count, stream));
    if (gws_total > 0) JSVD_CUDA_TRY(cudaMallocAsync(&d_ws, sizeof(double) * gws_total, stream));
    JSVD_CUDA_TRY(cudaMemcpyAsync(d_desc, ordered.data(), sizeof(BatchDesc) * ordered.size(), cudaMemcpyHostToDevice,
                                  stream));
    JSVD_CUDA_TRY(cudaMemsetAsync(d_next, 0, sizeof(int) * ngroups, stream));
    for (int c : {2, 3, 4})
        for (BatchRows rows : {kRowsAny, kRows256, kRows128})
            JSVD_CUDA_TRY(cudaFuncSetAttribute(batch_fn(c, rows), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem_cap));
    JSVD_CUDA_TRY(cudaEventRecord(ts->t0, stream));
    int launches = 0;
    std::vector<int> class_count(kClasses, 0);
    for (size_t k = 0; k < groups.size(); ++k) {
        const Group &g = groups[k];
        const int c = g.cls;
        // The classes run one after another on one stream: persistent CTAs of
        // a class hold their SMs until its queue drains, and concurrent classes
        // starved each other (a 512-thread CTA of the global class fills an
        // SM's register file).  The groups of a class, which are one class split
        // by kernel, overlap: each begins on the SMs that the one before leaves
        // (end_after_previous).  One after another, four members of class 2
        // between 100 and 300 rows took 8.6 ms, the longest alone 3.4.
        const bool first_of_class = k == 0 || groups[k - 1].cls != c;
        if (first_of_class) JSVD_CUDA_TRY(cudaEventRecord(ts->c0[c], stream));
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = first_of_class ? 0 : 1;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)g.grid);
        lc.stream = stream;
        lc.attrs = at;
        lc.numAttrs = 1;
        class_count[c] += g.count;
        if (g.csize > 0) {
            at[1].id = cudaLaunchAttributeClusterDimension;
            at[1].val.clusterDim.x = (unsigned)g.csize;
            at[1].val.clusterDim.y = 1;
            at[1].val.clusterDim.z = 1;
            lc.numAttrs = 2;
            lc.blockDim = dim3(g.share ? kClusterThreadsShared : kClusterThreads);
            lc.dynamicSmemBytes = g.smem;
            JSVD_CUDA_TRY(cudaLaunchKernelEx(&lc, cluster_fn(g.csize, g.tall, g.share), (const BatchDesc *)(d_desc + g.first), g.count,
                                             d_next + k, req.a, req.a_is_f32, req.eps, req.max_sweeps, req.sigma,
                                             req.v, req.u, d_sweeps + g.first));
        } else {
            const Class &cl = classes[c];
            // The global class keeps leading columns of A in the shared memory left over.
            const size_t dyn = (!cl.a_shared && !cl.v_shared) ? (smem_cap & ~(size_t)7) : g.smem;
            lc.blockDim = dim3((unsigned)g.threads);
            lc.dynamicSmemBytes = dyn;
            JSVD_CUDA_TRY(cudaLaunchKernelEx(&lc, batch_fn(c, g.rows), (const BatchDesc *)(d_desc + g.first), g.count,
                                             d_next + k, req.a, req.a_is_f32, req.eps, req.max_sweeps, req.sigma,
                                             req.v, req.u, d_sweeps + g.first, d_ws + gws_base[k], g.gws,
                                             (int)(dyn / sizeof(double))));
        }
        if (k + 1 == groups.size() || groups[k + 1].cls != c) JSVD_CUDA_TRY(cudaEventRecord(ts->c1[c], stream));
        ++launches;
    }
    JSVD_CUDA_TRY(cudaEventRecord(ts->t1, stream));
    std::vector<int> h_sweeps(count);
    JSVD_CUDA_TRY(cudaMemcpyAsync(h_sweeps.data(), d_sweeps, sizeof(int) * count, cudaMemcpyDeviceToHost, stream));
    JSVD_CUDA_TRY(cudaStreamSynchronize(stream));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ts->t0, ts->t1);
    BatchStats &st = batch_stats();
    st.calls += 1;
    st.launches += (unsigned long long)launches;
    st.kernel_ms += ms;
    unsigned long long total_sweeps = 0;
    for (int p = 0; p < count; ++p) {
        total_sweeps += (unsigned long long)h_sweeps[p];
        if (req.sweeps) req.sweeps[order_index[p]] = h_sweeps[p];
    }
    st.sweeps += total_sweeps;
    st.matrices += (unsigned long long)count;
    for (int c = 0; c < kClasses; ++c) {
        st.class_count[c] += (unsigned long long)class_count[c];
        float cms = 0.f;
        if (class_count[c] > 0 && cudaEventElapsedTime(&cms, ts->c0[c], ts->c1[c]) == cudaSuccess)
            st.class_ms[c] += cms;
    }
    return JSVD_OK;
}

}  // namespace jsvd

using namespace jsvd;

namespace jsvd {

size_t step_smem(int m, int n, bool v_shared)
{
    return sizeof(double) * (round_scratch_doubles(n) + (size_t)m * n + (v_shared ? (size_t)n * n : 0));
}

bool step_fits(int m, int n, size_t *smem_cap_out)
{
    int dev = 0;
    size_t cap = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || batch_smem_cap(dev, &cap) != JSVD_OK) return false;
    if (smem_cap_out) *smem_cap_out = cap;
    return step_smem(m, n, false) <= cap;
}

int StepScratch::ensure(int count)
{
    if (count <= cap) return JSVD_OK;
    if (d_descs) cudaFree(d_descs);
    if (d_rot) cudaFree(d_rot);
    if (h_rot) cudaFreeHost(h_rot);
    d_descs = nullptr;
    d_rot = nullptr;
    h_rot = nullptr;
    cap = 0;
    const int c = std::max(count, 256);
    JSVD_CUDA_TRY(cudaMalloc((void **)&d_descs, sizeof(StepDesc) * 2 * c));
    JSVD_CUDA_TRY(cudaMalloc((void **)&d_rot, sizeof(int) * c));
    JSVD_CUDA_TRY(cudaMallocHost((void **)&h_rot, sizeof(int) * c));
    cap = c;
    return JSVD_OK;
}

StepScratch::~StepScratch()
{
    if (d_descs) cudaFree(d_descs);
    if (d_rot) cudaFree(d_rot);
    if (h_rot) cudaFreeHost(h_rot);
}

int batch_step(const std::vector<StepDesc> &descs, double eps, int *rotated, StepScratch &sc, cudaStream_t st)
{
    const int count = (int)descs.size();
    if (count == 0) return JSVD_OK;
    int dev = 0;
    size_t cap = 0;
    JSVD_CUDA_TRY(cudaGetDevice(&dev));
    if (int rc = batch_smem_cap(dev, &cap); rc != JSVD_OK) return rc;
    if (int rc = sc.ensure(count); rc != JSVD_OK) return rc;
    // members whose V fits beside A in shared memory first, the others after
    std::vector<int> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_partition(order.begin(), order.end(),
                          [&](int i) { return step_smem(descs[i].m, descs[i].n, true) <= cap; });
    std::vector<StepDesc> sorted(count);
    size_t smem_vs = 0, smem_vg = 0;
    int n_vs = 0;
    for (int i = 0; i < count; ++i) {
        const StepDesc &d = descs[order[i]];
        sorted[i] = d;
        if (step_smem(d.m, d.n, true) <= cap) {
            smem_vs = std::max(smem_vs, step_smem(d.m, d.n, true));
            ++n_vs;
        } else {
            if (step_smem(d.m, d.n, false) > cap) return invalid_argument("A step member does not fit shared memory.");
            smem_vg = std::max(smem_vg, step_smem(d.m, d.n, false));
        }
    }
    JSVD_CUDA_TRY(cudaMemcpyAsync(sc.d_descs, sorted.data(), sizeof(StepDesc) * count, cudaMemcpyHostToDevice, st));
    static thread_local unsigned long long attr_done = 0;
    if (dev < 64 && !(attr_done & (1ull << dev))) {
        JSVD_CUDA_TRY(cudaFuncSetAttribute(batch_step_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)cap));
        JSVD_CUDA_TRY(cudaFuncSetAttribute(batch_step_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)cap));
        attr_done |= 1ull << dev;
    }
    if (n_vs > 0) batch_step_kernel<true><<<n_vs, 256, smem_vs, st>>>(sc.d_descs, eps, sc.d_rot);
    if (count > n_vs)
        batch_step_kernel<false><<<count - n_vs, 256, smem_vg, st>>>(sc.d_descs + n_vs, eps, sc.d_rot + n_vs);
    JSVD_CUDA_TRY(cudaGetLastError());
    JSVD_CUDA_TRY(cudaMemcpyAsync(sc.h_rot, sc.d_rot, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
    JSVD_CUDA_TRY(cudaStreamSynchronize(st));
    for (int i = 0; i < count; ++i) rotated[order[i]] = sc.h_rot[i];
    return JSVD_OK;
}

int batch_finish(const std::vector<StepDesc> &descs, double eps, StepScratch &sc, cudaStream_t st)
{
    const int count = (int)descs.size();
    if (count == 0) return JSVD_OK;
    if (int rc = sc.ensure(count); rc != JSVD_OK) return rc;
    StepDesc *d2 = sc.d_descs + sc.cap;  // the second half: the step's descriptors may still be read
    JSVD_CUDA_TRY(cudaMemcpyAsync(d2, descs.data(), sizeof(StepDesc) * count, cudaMemcpyHostToDevice, st));
    batch_finish_kernel<<<count, 256, 0, st>>>(d2, eps);
    JSVD_CUDA_TRY(cudaGetLastError());
    return JSVD_OK;
}

}  // namespace jsvd

using namespace jsvd;

extern "C" int jsvd_batch_svd_device(int count, const int *rows, const int *cols, const long long *a_offsets,
                                     const void *d_a, int a_is_f32, const jsvd_config *cfg, double *d_sigma,
                                     double *d_v, double *d_u, int *sweeps, const jsvd_batch_tuning *tuning,
                                     void *stream)
{
    return c_entry([&]() -> int {
        set_last_error(JSVD_OK, "");
        jsvd_config def;
        const jsvd_config &c = config_or_default(cfg, def);
        const int bad = check_batch_args(count, rows, cols, a_offsets, d_a, d_sigma == nullptr, c);
        if (bad != JSVD_OK) return bad;
        if (count == 0) return JSVD_OK;  // nothing to solve, no CUDA call
        cudaStream_t st = nullptr;
        if (const int e = entry_stream(stream, &st); e != JSVD_OK) return e;
        BatchRequest req;
        req.count = count;
        req.rows = rows;
        req.cols = cols;
        req.a_offsets = a_offsets;
        req.a = d_a;
        req.a_is_f32 = a_is_f32;
        req.eps = c.epsilon;
        req.max_sweeps = c.max_sweeps;
        req.sigma = d_sigma;
        req.v = d_v;
        req.u = d_u;
        req.sweeps = sweeps;
        req.tuning = tuning;
        return batch_solve(req, st);
    });
}

extern "C" void jsvd_batch_stats_get(jsvd_batch_stats *out)
{
    if (!out) return;
    const BatchStats &s = batch_stats();
    out->calls = s.calls;
    out->launches = s.launches;
    out->matrices = s.matrices;
    out->sweeps = s.sweeps;
    out->kernel_ms = s.kernel_ms;
    for (int c = 0; c < 5; ++c) {
        out->class_count[c] = s.class_count[c];
        out->class_ms[c] = s.class_ms[c];
    }
}

extern "C" void jsvd_batch_stats_reset(void) { batch_stats() = BatchStats{}; }

extern "C" int jsvd_batch_set_cluster_classes(int mask, int *previous)
{
    if (mask & ~((1 << 2) | (1 << 3) | (1 << 4)))
        return invalid_argument("Only size classes 2, 3 and 4 can be solved by clusters.");
    const int old = g_cluster_mask.exchange(mask);
    if (previous) *previous = old;
    return JSVD_OK;
}

extern "C" void jsvd_batch_builtin_tuning(jsvd_batch_tuning *out)
{
    if (!out) return;
    for (int c = 0; c < kClasses; ++c) out[c] = kBuiltinTuning[c];
}

namespace jsvd {
namespace {

// Candidate launch shapes of class c whose largest sampled member needs
// smem_need bytes of shared memory.  Classes 0-2: threads x persistent CTAs
// per SM, as many CTAs as the SM's shared memory and 2048 threads allow.
// Classes 3-4 take a whole SM's shared memory per CTA: threads x grid cap
// (the cap bounds the per-CTA global-memory slices that compete for L2).
std::vector<jsvd_batch_tuning> batch_candidates(int c, size_t smem_need, int sms, size_t smem_per_sm)
{
    std::vector<jsvd_batch_tuning> out;
    for (int t : {128, 256, 512}) {
        if (c <= 2) {
            for (int k : {1, 2, 4, 8})
                if (t * k <= 2048 && (size_t)k * (smem_need + 1024) <= smem_per_sm) out.push_back({t, k, 0});
        } else {
            for (int cap : {0, (3 * sms) / 4, sms / 2}) out.push_back({t, 1, cap});
        }
    }
    return out;
}

bool same_shape(const jsvd_batch_tuning &x, const jsvd_batch_tuning &y)
{
    return x.threads == y.threads && x.ctas_per_sm == y.ctas_per_sm && x.max_ctas == y.max_ctas;
}

}  // namespace
}  // namespace jsvd

extern "C" int jsvd_batch_autotune(int count, const int *rows, const int *cols, const long long *a_offsets,
                                   const void *d_a, int a_is_f32, const jsvd_config *cfg, int sample, int reps,
                                   int want_u, int want_v, jsvd_batch_autotune_report *report, void *stream)
{
    return c_entry([&]() -> int {
        set_last_error(JSVD_OK, "");
        jsvd_config def;
        const jsvd_config &c = config_or_default(cfg, def);
        if (report == nullptr) return invalid_argument("Autotune report must not be null.");
        const int bad = check_batch_args(count, rows, cols, a_offsets, d_a, false, c);
        if (bad != JSVD_OK) return bad;
        *report = jsvd_batch_autotune_report{};
        for (int k = 0; k < kClasses; ++k) report->builtin[k] = kBuiltinTuning[k];
        if (count == 0) return JSVD_OK;
        if (reps <= 0) reps = 2;
        cudaStream_t st = nullptr;
        if (const int e = entry_stream(stream, &st); e != JSVD_OK) return e;
        int dev = 0;
        JSVD_CUDA_TRY(cudaGetDevice(&dev));
        int sms = 0, smem_per_sm = 0;
        JSVD_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        JSVD_CUDA_TRY(cudaDeviceGetAttribute(&smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
        size_t smem_cap = 0;
        int rc = batch_smem_cap(dev, &smem_cap);
        if (rc != JSVD_OK) return rc;

        std::vector<std::vector<int>> members(kClasses);
        for (int i = 0; i < count; ++i) {
            if (rows[i] <= 0 || cols[i] <= 0 || rows[i] < cols[i])
                return invalid_argument("Batch matrix shape must satisfy rows >= columns > 0.");
            if (dims_out_of_range((size_t)rows[i], (size_t)cols[i])) {
                set_last_error(JSVD_ERR_OVERFLOW, "Matrix dimensions exceed the supported range.");
                return JSVD_ERR_OVERFLOW;
            }
            members[member_class(rows[i], cols[i], smem_cap, nullptr)].push_back(i);
        }

        // Flush buffer (larger than L2) and output buffers sized for the largest sample.
        const size_t flush_bytes = (size_t)256 << 20;
        std::vector<std::vector<int>> picked(kClasses);
        size_t max_s = 0, max_v = 0, max_u = 0;
        for (int k = 0; k < kClasses; ++k) {
            auto &mem = members[k];
            std::sort(mem.begin(), mem.end(),
                      [&](int x, int y) { return member_work(rows[x], cols[x]) > member_work(rows[y], cols[y]); });
            const size_t cnt = mem.size();
            const size_t s = (sample > 0 && (size_t)sample < cnt) ? (size_t)sample : cnt;
            size_t ns = 0, nv = 0, nu = 0;
            for (size_t j = 0; j < s; ++j) {  // evenly spaced over the work order
                const int i = mem[j * cnt / s];
                picked[k].push_back(i);
                ns += (size_t)cols[i];
                nv += (size_t)cols[i] * cols[i];
                nu += (size_t)rows[i] * cols[i];
            }
            max_s = std::max(max_s, ns);
            max_v = std::max(max_v, nv);
            max_u = std::max(max_u, nu);
            report->members[k] = (int)cnt;
            report->sampled[k] = (int)s;
        }
        void *d_flush = nullptr;
        double *d_sigma = nullptr, *d_v = nullptr, *d_u = nullptr;
        // The autotuner's own solves are not counted in the batch statistics.
        // Buffers and statistics are restored on every path, a C++ exception's
        // included.
        const BatchStats saved = batch_stats();
        ScopeExit restore([&] {
            if (d_flush) cudaFreeAsync(d_flush, st);
            if (d_sigma) cudaFreeAsync(d_sigma, st);
            if (d_v) cudaFreeAsync(d_v, st);
            if (d_u) cudaFreeAsync(d_u, st);
            cudaStreamSynchronize(st);
            batch_stats() = saved;
        });
        if (cudaMallocAsync(&d_flush, flush_bytes, st) != cudaSuccess ||
            cudaMallocAsync((void **)&d_sigma, sizeof(double) * std::max<size_t>(max_s, 1), st) != cudaSuccess ||
            (want_v &&
             cudaMallocAsync((void **)&d_v, sizeof(double) * std::max<size_t>(max_v, 1), st) != cudaSuccess) ||
            (want_u && cudaMallocAsync((void **)&d_u, sizeof(double) * std::max<size_t>(max_u, 1), st) != cudaSuccess))
            return cuda_failure(cudaGetLastError(), "cudaMallocAsync", __FILE__, __LINE__);

        for (int k = 0; k < kClasses; ++k) {
            const auto &pk = picked[k];
            if (pk.empty()) continue;
            const int s = (int)pk.size();
            std::vector<int> r_s(s), c_s(s), sw(s), sw_ref(s);
            std::vector<long long> off_s(s);
            size_t need = 0, nsig = 0;
            for (int j = 0; j < s; ++j) {
                r_s[j] = rows[pk[j]];
                c_s[j] = cols[pk[j]];
                off_s[j] = a_offsets[pk[j]];
                size_t nj = 0;
                member_class(r_s[j], c_s[j], smem_cap, &nj);
                need = std::max(need, nj);
                nsig += (size_t)c_s[j];
            }
            std::vector<double> sig(nsig), sig_ref(nsig);
            // the built-in shape first: it is the yardstick and the bitwise reference
            std::vector<jsvd_batch_tuning> cands{kBuiltinTuning[k]};
            for (const auto &t : batch_candidates(k, need, sms, (size_t)smem_per_sm))
                if (!same_shape(t, kBuiltinTuning[k])) cands.push_back(t);
            report->candidates[k] = (int)cands.size();
            double best_ms = -1.0;
            jsvd_batch_tuning best = kBuiltinTuning[k];
            for (size_t ci = 0; ci < cands.size(); ++ci) {
                jsvd_batch_tuning tun[kClasses] = {};
                tun[k] = cands[ci];
                BatchRequest req;
                req.count = s;
                req.rows = r_s.data();
                req.cols = c_s.data();
                req.a_offsets = off_s.data();
                req.a = d_a;
                req.a_is_f32 = a_is_f32;
                req.eps = c.epsilon;
                req.max_sweeps = c.max_sweeps;
                req.sigma = d_sigma;
                req.v = d_v;
                req.u = d_u;
                req.sweeps = sw.data();
                req.tuning = tun;
                double ms = -1.0;
                for (int r = 0; r < reps; ++r) {
                    if (cudaMemsetAsync(d_flush, r & 0xff, flush_bytes, st) != cudaSuccess)
                        return cuda_failure(cudaGetLastError(), "cudaMemsetAsync", __FILE__, __LINE__);
                    const double before = batch_stats().class_ms[k];
                    rc = batch_solve(req, st);
                    if (rc != JSVD_OK) return rc;
                    const double t = batch_stats().class_ms[k] - before;
                    ms = ms < 0.0 ? t : std::min(ms, t);
                }
                if (cudaMemcpyAsync(sig.data(), d_sigma, sizeof(double) * nsig, cudaMemcpyDeviceToHost, st) !=
                        cudaSuccess ||
                    cudaStreamSynchronize(st) != cudaSuccess)
                    return cuda_failure(cudaGetLastError(), "cudaMemcpyAsync", __FILE__, __LINE__);
                if (ci == 0) {
                    sig_ref = sig;
                    sw_ref = sw;
                    report->builtin_ms[k] = ms;
                } else if (std::memcmp(sig.data(), sig_ref.data(), sizeof(double) * nsig) != 0 || sw != sw_ref) {
                    set_last_error(JSVD_ERR_RUNTIME, "Batch launch shapes disagree on sigma or sweep counts.");
                    return JSVD_ERR_RUNTIME;
                }
                if (best_ms < 0.0 || ms < best_ms) {
                    best_ms = ms;
                    best = cands[ci];
                }
            }
            // a shape replaces the built-in one only when it is more than 2% faster
            if (best_ms > 0.98 * report->builtin_ms[k]) {
                best = kBuiltinTuning[k];
                best_ms = report->builtin_ms[k];
            }
            report->best[k] = best;
            report->best_ms[k] = best_ms;
        }
        return JSVD_OK;
    });
}
