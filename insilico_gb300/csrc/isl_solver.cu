// Krylov solve of the assembled system on the GB300.
//
// Jacobi-preconditioned CG with the semantics of Eigen 3.2's
// ConjugateGradient<SparseMatrix<double>> as the reference calls it
// (base/solver/Eigen3.hpp:265-275): x0 = 0, z = D^{-1} r, stop when
// ||r||^2 < tol^2 ||b||^2 or after max_iter iterations.
//
// One iteration = three kernels on the context stream:
//   k_cg_dir   : p = D^{-1} r + beta p          (beta = 0 on the first pass)
//   k_spmv_pap : q = A p and p.q                (last block: alpha)
//   k_cg_update: x += alpha p, r -= alpha q,  r.r and r.D^{-1}r
//                                               (last block: convergence, beta)
// Block partial sums are reduced by the last block to finish (a ticket
// counter orders the blocks; no atomics touch the data), in a fixed order, so
// results are bit-reproducible.  CHUNK iterations are captured once into a
// CUDA graph that is replayed until the device-side done flag is set.
//
// The mixed method is CG in FP32 (vectors and matrix values; dot products
// reduced in FP64) with reliable updates in FP64: whenever the iterated FP32
// residual has dropped by a factor 10 since the last update (or has met the
// tolerance), the FP32 increment is folded into the FP64 iterate, the true
// residual r = b - A64 x is formed in FP64 and replaces the iterated one, and
// the iteration continues with the same search direction.  The solve ends
// when the true FP64 residual meets the tolerance.
#include <cmath>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "isl_coarse.h"
#include "isl_internal.h"
#include "isl_device.cuh"

namespace isl {

constexpr int BS = 256;
constexpr int CHUNK = 32;
// reliable update when the iterated residual has dropped 10x (squared: 1e-2);
// the one-cluster solve of small systems uses this, the graph paths the
// context's ISL_OPT_RELIABLE_DROP (default the same)
constexpr double kDelta2 = 1e-2;

// q = A p; partial p.q; last block: alpha = absNew / p.q
template <typename TV, typename TX, int LPR>
__global__ void __launch_bounds__(BS) k_spmv_pap(int n, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                                 const TV* __restrict__ val, const TX* __restrict__ p, TX* __restrict__ q,
                                                 CGScal* S, double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const int lane = threadIdx.x % LPR;
    const int grp = (blockIdx.x * BS + threadIdx.x) / LPR, ngrp = gridDim.x * BS / LPR;
    const int wgrp = grp - grp % (32 / LPR);  // first group of this warp: the loop is warp-uniform
    TX loc = TX(0);  // accumulated in the vectors' precision, summed across warps in FP64
    for (int base = wgrp; base < n; base += ngrp) {
        const int row = base + (grp - wgrp);
        const bool act = row < n;
        const TX acc = row_dot<TV, TX, LPR>(row, act, rowptr, colind, val, p, lane);
        if (act && lane == 0) {
            q[row] = acc;
            loc += p[row] * acc;
        }
    }
    double tot = 0.0;
    bool last;
    if constexpr (std::is_same<TX, float>::value) {  // FP32 vectors: double-float block and grid sums
        const df bs = block_sum_df(loc, reinterpret_cast<float*>(sh));
        if (threadIdx.x == 0) reinterpret_cast<float2*>(part)[blockIdx.x] = make_float2(bs.hi, bs.lo);
        last = last_block(&S->ticket1);
        if (last) tot = reduce_parts_df_blk<BS>(reinterpret_cast<const float2*>(part), gridDim.x, sh);
    } else {
        const double bs = block_sum_t(loc, sh);
        if (threadIdx.x == 0) part[blockIdx.x] = bs;
        last = last_block(&S->ticket1);
        if (last) tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
    }
    if (last && threadIdx.x == 0) {
        S->pAp = tot;
        S->alpha = S->absNew / tot;
        S->ticket1 = 0;
    }
}

// x += alpha p; r -= alpha q; partial r.r, r.z; last block: convergence + beta
template <typename TX>
__global__ void __launch_bounds__(BS) k_cg_update(int n, TX* __restrict__ x, TX* __restrict__ r, const TX* __restrict__ p,
                                                  const TX* __restrict__ q, const TX* __restrict__ dinv, CGScal* S,
                                                  double* part, int max_iter) {
    if (S->done) return;
    __shared__ double sh[32];
    const TX alpha = (TX)S->alpha;
    TX rr = TX(0), rz = TX(0);
    const int stride = gridDim.x * BS;
    int i = blockIdx.x * BS + threadIdx.x;
    // four entries per pass, loads issued together: the grid is small (see
    // upd_grid), so each thread keeps several loads in flight
    for (; i + 3 * stride < n; i += 4 * stride) {
        TX pv[4], qv[4], rv[4], dv[4], xv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            pv[k] = ld(p + i + k * stride); qv[k] = ld(q + i + k * stride); dv[k] = ld(dinv + i + k * stride);
            rv[k] = r[i + k * stride]; xv[k] = x[i + k * stride];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[i + k * stride] = xv[k] + alpha * pv[k];
            const TX ri = rv[k] - alpha * qv[k];
            r[i + k * stride] = ri;
            rr += ri * ri;
            rz += ri * (dv[k] * ri);
        }
    }
    for (; i < n; i += stride) {
        x[i] += alpha * p[i];
        const TX ri = r[i] - alpha * q[i];
        r[i] = ri;
        rr += ri * ri;
        rz += ri * (dinv[i] * ri);
    }
    bool last;
    double trr = 0.0, trz = 0.0;
    if constexpr (std::is_same<TX, float>::value) {  // FP32 vectors: double-float block and grid sums
        df b1, b2;
        block_sum_df2(rr, rz, reinterpret_cast<float*>(sh), b1, b2);
        if (threadIdx.x == 0) reinterpret_cast<float4*>(part)[blockIdx.x] = make_float4(b1.hi, b1.lo, b2.hi, b2.lo);
        last = last_block(&S->ticket2);
        if (last) reduce_parts2_df_blk<BS>(reinterpret_cast<const float4*>(part), gridDim.x, sh, trr, trz);
    } else {
        const double b1 = block_sum_t(rr, sh);
        const double b2 = block_sum_t(rz, sh);
        if (threadIdx.x == 0) { part[2 * blockIdx.x] = b1; part[2 * blockIdx.x + 1] = b2; }
        last = last_block(&S->ticket2);
        if (last) reduce_parts2_blk<BS>(part, gridDim.x, sh, trr, trz);
    }
    if (last) {
        if (threadIdx.x == 0) {
            S->rr = trr;
            S->iters += 1;
            S->absOld = S->absNew;
            S->beta = trz / S->absNew;
            S->absNew = trz;
            if (!(trr == trr) || !(trz == trz)) { S->bad = 1; S->done = 1; }
            else if (trr < S->threshold) S->done = 1;
            else if (trr < S->rrtrig) S->done = 3;
            else if (S->iters >= max_iter) S->done = 2;
            S->ticket2 = 0;
        }
    }
}

template <typename TX>
__global__ void __launch_bounds__(BS) k_cg_dir(int n, const TX* __restrict__ r, const TX* __restrict__ dinv, TX* __restrict__ p,
                                               const CGScal* S) {
    if (S->done) return;
    const TX beta = (TX)S->beta;
    for (int i = blockIdx.x * BS + threadIdx.x; i < n; i += gridDim.x * BS) p[i] = dinv[i] * r[i] + beta * p[i];
}

// x = 0, r = b, p = 0, beta = 0, absNew = r.D^{-1}r, rhsNorm2 = b.b (FP64)
template <typename TB, typename TX>
__global__ void __launch_bounds__(BS) k_cg_init(int n, const TB* __restrict__ b, TX* __restrict__ x, TX* __restrict__ r,
                                                TX* __restrict__ p, const TX* __restrict__ dinv, CGScal* S, double* part,
                                                double tol, double trig) {
    __shared__ double sh[32];
    double bb = 0.0, bz = 0.0;
    for (int i = blockIdx.x * BS + threadIdx.x; i < n; i += gridDim.x * BS) {
        const TB bi = b[i];
        const TX ri = (TX)bi;
        x[i] = TX(0);
        r[i] = ri;
        p[i] = TX(0);
        bb += (double)bi * (double)bi;
        bz += (double)ri * (double)(dinv[i] * ri);
    }
    const double b1 = block_sum(bb, sh);
    const double b2 = block_sum(bz, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = b1; part[2 * blockIdx.x + 1] = b2; }
    if (last_block(&S->ticket2)) {
        double tbb, tbz;
        reduce_parts2(part, gridDim.x, sh, tbb, tbz);
        if (threadIdx.x == 0) {
            S->rhsNorm2 = tbb;
            S->threshold = tol * tol * tbb;
            S->rrtrig = trig * tbb;
            S->absNew = tbz;
            S->absOld = tbz;
            S->beta = 0.0;
            S->rr = tbb;
            S->iters = 0;
            S->bad = !(tbb == tbb);
            S->done = (tbb == 0.0 || tbb < S->threshold || S->bad) ? 1 : 0;
            S->ticket1 = 0;
            S->ticket2 = 0;
        }
    }
}

template <typename TV, typename TX>
__global__ void k_dinv(int n, const int* __restrict__ diag, const TV* __restrict__ val, TX* __restrict__ dinv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const TV d = val[diag[i]];
        dinv[i] = (d != TV(0)) ? TX(1) / (TX)d : TX(1);
    }
}

// reliable update, part 1: fold the FP32 increment into the FP64 iterate
__global__ void k_fold(int n, float* __restrict__ x32, double* __restrict__ x64) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        x64[i] += (double)x32[i];
        x32[i] = 0.0f;
    }
}

// r64 = b - A64 x64 ; last block: ||r64||^2 -> *out
template <int LPR>
__global__ void __launch_bounds__(BS) k_residual64(int n, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                                   const double* __restrict__ val, const double* __restrict__ x,
                                                   const double* __restrict__ b, double* __restrict__ r, double* part,
                                                   unsigned int* ticket, double* out) {
    __shared__ double sh[32];
    const int lane = threadIdx.x % LPR;
    const int grp = (blockIdx.x * BS + threadIdx.x) / LPR, ngrp = gridDim.x * BS / LPR;
    const int wgrp = grp - grp % (32 / LPR);
    double loc = 0.0;
    for (int base = wgrp; base < n; base += ngrp) {
        const int row = base + (grp - wgrp);
        const bool act = row < n;
        const double ax = row_dot<double, double, LPR>(row, act, rowptr, colind, val, x, lane);
        if (act && lane == 0) {
            const double ri = b[row] - ax;
            r[row] = ri;
            loc += ri * ri;
        }
    }
    const double bs = block_sum(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bs;
    if (last_block(ticket)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) { *out = tot; *ticket = 0; }
    }
}

// reliable update, part 2: r32 = r64; beta = (r.z)_new / (r.z)_previous; resume
// fresh != 0: the true residual has not dropped since the previous reliable
// update, so the FP32 directions have lost conjugacy: restart them (beta = 0)
__global__ void __launch_bounds__(BS) k_restart32(int n, const double* __restrict__ r64, float* __restrict__ r32,
                                                  const float* __restrict__ dinv, CGScal* S, double* part, double rrtrig,
                                                  int fresh) {
    __shared__ double sh[32];
    double rr = 0.0, rz = 0.0;
    for (int i = blockIdx.x * BS + threadIdx.x; i < n; i += gridDim.x * BS) {
        const float ri = (float)r64[i];
        r32[i] = ri;
        rr += (double)ri * (double)ri;
        rz += (double)ri * (double)(dinv[i] * ri);
    }
    const double b1 = block_sum(rr, sh);
    const double b2 = block_sum(rz, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = b1; part[2 * blockIdx.x + 1] = b2; }
    if (last_block(&S->ticket2)) {
        double trr, trz;
        reduce_parts2_blk<BS>(part, gridDim.x, sh, trr, trz);
        if (threadIdx.x == 0) {
            S->rr = trr;
            S->beta = fresh ? 0.0 : trz / S->absOld;
            S->absNew = trz;
            S->rrtrig = rrtrig;
            S->done = 0;
            S->ticket2 = 0;
        }
    }
}

__global__ void k_copy64(int n, const double* __restrict__ a, double* __restrict__ b) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = a[i];
}

// ---------------------------------------------------------------------------
static unsigned vec_grid(isl_ctx* c) { return (unsigned)c->sm_count * (2048 / BS); }
// grid of the CG update kernels: two blocks per SM keep the reduction tail
// (one partial per block, last-block ticket) short
static unsigned upd_grid(const isl_ctx* c, long long n) {
    return (unsigned)std::max<long long>(1, std::min<long long>((n + BS - 1) / BS, 2LL * c->sm_count));
}

template <typename TV, typename TX>
static void launch_spmv(int lpr, unsigned grid, cudaStream_t st, int n, const int* rp, const int* ci, const TV* v, const TX* p,
                        TX* q, CGScal* S, double* part) {
    switch (lpr) {
        case 2: k_spmv_pap<TV, TX, 2><<<grid, BS, 0, st>>>(n, rp, ci, v, p, q, S, part); break;
        case 4: k_spmv_pap<TV, TX, 4><<<grid, BS, 0, st>>>(n, rp, ci, v, p, q, S, part); break;
        case 8: k_spmv_pap<TV, TX, 8><<<grid, BS, 0, st>>>(n, rp, ci, v, p, q, S, part); break;
        case 16: k_spmv_pap<TV, TX, 16><<<grid, BS, 0, st>>>(n, rp, ci, v, p, q, S, part); break;
        default: k_spmv_pap<TV, TX, 32><<<grid, BS, 0, st>>>(n, rp, ci, v, p, q, S, part); break;
    }
}

static void launch_residual(int lpr, unsigned grid, cudaStream_t st, int n, const int* rp, const int* ci, const double* v,
                            const double* x, const double* b, double* r, double* part, unsigned* ticket, double* out) {
    switch (lpr) {
        case 2: k_residual64<2><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, part, ticket, out); break;
        case 4: k_residual64<4><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, part, ticket, out); break;
        case 8: k_residual64<8><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, part, ticket, out); break;
        case 16: k_residual64<16><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, part, ticket, out); break;
        default: k_residual64<32><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, part, ticket, out); break;
    }
}

// q = A p and p.q on the scalar sliced-ELL copy (one warp per slice of 32
// sorted rows, one lane per row).  The loads of U slots (column id and value,
// 128 coalesced bytes per warp each, L1 bypassed) are issued before their U
// gathers of p, so every lane keeps 8U bytes of the stream in flight; the
// FMAs then run in slot order, so the sums do not depend on U.  Padding slots
// hold value 0 and a valid column.  The stream is latency-bound: the variants
// run at full occupancy (U = 2, 4: 8 blocks of 256 per SM within 32
// registers; U = 8: 6 blocks), which measured faster on the GB300 than deeper
// batches at lower occupancy.
// TC = short: each slot holds its column as a 16-bit offset from the lane's
// row (row 0 for a padding lane), 6 B per stored entry instead of 8
template <int U, int MINB, typename TC>
__global__ void __launch_bounds__(BS, MINB) k_sspmv_batch(int nslice, const int* __restrict__ soff,
                                                          const int* __restrict__ swid, const int* __restrict__ srow,
                                                          const TC* __restrict__ scol, const float* __restrict__ sv,
                                                          const float* __restrict__ p, float* __restrict__ q, CGScal* S,
                                                          double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * BS + threadIdx.x) >> 5, nwarps = gridDim.x * (BS / 32);
    float loc = 0.f;
    for (int s = warp; s < nslice; s += nwarps) {
        const int o = soff[s] + lane, w = swid[s];  // w: warp-uniform
        const int row = srow[s * 32 + lane];
        const int base = sizeof(TC) == 2 ? max(row, 0) : 0;
        float acc = 0.f;
        for (int k = 0; k < w; k += U) {
            int j[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u < w) {
                    j[u] = ld_stream(scol + o + (k + u) * 32) + base;
                    v[u] = ld_stream(sv + o + (k + u) * 32);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + u < w) acc += v[u] * __ldg(p + j[u]);
        }
        if (row >= 0) {
            q[row] = acc;
            loc += p[row] * acc;
        }
    }
    const df bsum = block_sum_df(loc, reinterpret_cast<float*>(sh));
    if (threadIdx.x == 0) reinterpret_cast<float2*>(part)[blockIdx.x] = make_float2(bsum.hi, bsum.lo);
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_df_blk<BS>(reinterpret_cast<const float2*>(part), gridDim.x, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

static unsigned ssell_grid(const isl_ctx* c, unsigned per_sm) {
    const long long need = (c->ss_nslice + (BS / 32) - 1) / (BS / 32);
    return (unsigned)std::max<long long>(1, std::min<long long>(need, (long long)per_sm * c->sm_count));
}

// FP32 SpMV of the mixed solver: kind 2..32 = CSR with that many lanes per
// row, kind 100 + U = the sliced-ELL copy with U slots of loads in flight
static void launch_spmv32(isl_ctx* c, int kind, unsigned grid, cudaStream_t st, const float* p, float* q, CGScal* S,
                          double* part) {
    const int ns = (int)c->ss_nslice;
    const bool s16 = c->ss16 && c->use_scol16;  // 16-bit column offsets
    switch (kind) {
        case 102:
            if (s16) k_sspmv_batch<2, 8, short><<<ssell_grid(c, 8), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col16.p, c->dss_val.p, p, q, S, part);
            else k_sspmv_batch<2, 8, int><<<ssell_grid(c, 8), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col.p, c->dss_val.p, p, q, S, part);
            break;
        case 104:
            if (s16) k_sspmv_batch<4, 8, short><<<ssell_grid(c, 8), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col16.p, c->dss_val.p, p, q, S, part);
            else k_sspmv_batch<4, 8, int><<<ssell_grid(c, 8), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col.p, c->dss_val.p, p, q, S, part);
            break;
        case 108:
            if (s16) k_sspmv_batch<8, 6, short><<<ssell_grid(c, 6), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col16.p, c->dss_val.p, p, q, S, part);
            else k_sspmv_batch<8, 6, int><<<ssell_grid(c, 6), BS, 0, st>>>(ns, c->dss_off.p, c->dss_wid.p, c->dss_row.p, c->dss_col.p, c->dss_val.p, p, q, S, part);
            break;
        default: launch_spmv<float, float>(kind, grid, st, (int)c->neq, c->drowptr.p, c->dcolind.p, c->dval32.p, p, q, S, part); break;
    }
}

bool spmv32_kind_valid(const isl_ctx* c, int kind) {
    if (kind == 0 || kind == 2 || kind == 4 || kind == 8 || kind == 16 || kind == 32) return true;
    // a batch builds its sliced-ELL copy at its first mixed solve (and, should
    // the copy not fit 32-bit slot offsets, autotunes the CSR kernels instead)
    const bool batched = c->ninst > 1 || c->force_batched;
    return (kind == 102 || kind == 104 || kind == 108) && (c->ss_nslice > 0 || batched);
}

// FP32 values into the scalar sliced-ELL slots (padding slots stay zero)
__global__ void k_ssell_values(int n, const int* __restrict__ rowptr, const int* __restrict__ spos,
                               const float* __restrict__ val, float* __restrict__ sv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int lo = rowptr[i], hi = rowptr[i + 1], s0 = spos[i];
        for (int k = lo; k < hi; ++k) sv[s0 + (k - lo) * 32] = val[k];
    }
}

// refresh the sliced-ELL values after an assembly
int ensure_ssell(isl_ctx* c) {
    if (c->ss_nslice == 0 || c->ss_serial == c->asm_serial) return ISL_OK;
    k_ssell_values<<<vec_grid(c), BS, 0, c->stream>>>((int)c->neq, c->drowptr.p, c->dss_pos.p, c->dval32.p, c->dss_val.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 1;
    c->ss_serial = c->asm_serial;
    return ISL_OK;
}

// Autotune of the FP32 SpMV: CSR lanes per row and, when the sliced-ELL copy
// exists, its batch depths; each candidate timed over 20 launches on the
// current matrix, the fastest kept.  Chosen once per context.
static int autotune_spmv32(isl_ctx* c, const float* p, float* q, CGScal* S, double* part) {
    if (c->spmv32_forced && spmv32_kind_valid(c, c->spmv32_forced)) return c->spmv32_forced;
    const double avg = (double)c->nnz / (double)c->neq;
    int best = 2;
    while (best < 32 && best < avg / 2) best *= 2;
    if (c->neq < 20000) return best;  // too small to time meaningfully
    int cached = 0;
    if (tune_lookup(c, "spmv32", &cached) && spmv32_kind_valid(c, cached)) return cached;
    // preference order; the first within 2 % of the fastest is kept, so that
    // the choice (and the rounding of p.q, which follows the grid) does not
    // flip with timing noise
    int cand[7] = {104, 102, 108, 4, 8, 16, 32};
    if (c->ss_nslice == 0) { cand[0] = 4; cand[1] = 8; cand[2] = 16; cand[3] = 32; }
    const int ncand = c->ss_nslice > 0 ? 7 : 4;
    float ms_of[7];
    float bestms = 1e30f;
    cudaMemsetAsync(S, 0, sizeof(CGScal), c->stream);
    c->launches += 21 * ncand;
    for (int k = 0; k < ncand; ++k) {
        launch_spmv32(c, cand[k], vec_grid(c), c->stream, p, q, S, part);
        cudaEventRecord(c->ev[2], c->stream);
        for (int r = 0; r < 20; ++r) launch_spmv32(c, cand[k], vec_grid(c), c->stream, p, q, S, part);
        cudaEventRecord(c->ev[3], c->stream);
        cudaEventSynchronize(c->ev[3]);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev[2], c->ev[3]);
        ms_of[k] = ms;
        bestms = std::min(bestms, ms);
    }
    for (int k = 0; k < ncand; ++k)
        if (ms_of[k] <= 1.02f * bestms) { best = cand[k]; break; }
    tune_store(c, "spmv32", best);
    return best;
}

// Autotune of the SpMV row mapping (lanes per row): time each candidate on the
// current matrix, keep the fastest.  Chosen once per context and precision.
template <typename TV, typename TX>
static int autotune_lpr(isl_ctx* c, const TV* val, const TX* p, TX* q, CGScal* S, double* part) {
    const double avg = (double)c->nnz / (double)c->neq;
    int best = 2;
    while (best < 32 && best < avg / 2) best *= 2;
    if (c->neq < 20000) return best;  // too small to time meaningfully
    const char* tuner = sizeof(TV) == 8 ? "spmv64" : "spmv32csr";
    int cached = 0;
    if (tune_lookup(c, tuner, &cached) && (cached == 4 || cached == 8 || cached == 16 || cached == 32)) return cached;
    const int cand[4] = {4, 8, 16, 32};
    float bestms = 1e30f;
    cudaMemsetAsync(S, 0, sizeof(CGScal), c->stream);
    c->launches += 24;
    for (int k = 0; k < 4; ++k) {
        const int lpr = cand[k];
        launch_spmv<TV, TX>(lpr, vec_grid(c), c->stream, (int)c->neq, c->drowptr.p, c->dcolind.p, val, p, q, S, part);
        cudaEventRecord(c->ev[2], c->stream);
        for (int r = 0; r < 5; ++r)
            launch_spmv<TV, TX>(lpr, vec_grid(c), c->stream, (int)c->neq, c->drowptr.p, c->dcolind.p, val, p, q, S, part);
        cudaEventRecord(c->ev[3], c->stream);
        cudaEventSynchronize(c->ev[3]);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev[2], c->ev[3]);
        if (ms < bestms) { bestms = ms; best = lpr; }
    }
    tune_store(c, tuner, best);
    return best;
}

// one CHUNK of iterations (dir, spmv, update) captured into a graph
template <typename TV, typename TX>
static int capture_chunk(isl_ctx* c, const TV* val, TX* x, TX* r, TX* p, TX* q, const TX* dinv, int lpr, int max_iter,
                         cudaGraphExec_t* exec) {
    cudaStream_t st = c->stream;
    const int n = (int)c->neq;
    const unsigned grid = vec_grid(c);
    CGScal* S = c->dscal.p;
    double* part = c->dpart.p;
    cudaGraph_t graph;
    ISL_CHECK_CUDA(c, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    // the direction update has no reduction: one thread per entry, full grid
    const unsigned gdir = (unsigned)std::max<long long>(1, ((long long)n + BS - 1) / BS);
    for (int k = 0; k < CHUNK; ++k) {
        k_cg_dir<TX><<<gdir, BS, 0, st>>>(n, r, dinv, p, S);
        if constexpr (std::is_same<TV, float>::value)
            launch_spmv32(c, lpr, grid, st, p, q, S, part);
        else
            launch_spmv<TV, TX>(lpr, grid, st, n, c->drowptr.p, c->dcolind.p, val, p, q, S, part);
        k_cg_update<TX><<<upd_grid(c, n), BS, 0, st>>>(n, x, r, p, q, dinv, S, part, max_iter);
    }
    ISL_CHECK_CUDA(c, cudaStreamEndCapture(st, &graph));
    cudaError_t e = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    ISL_CHECK_CUDA(c, e);
    return ISL_OK;
}

cudaError_t grid_barrier_start(isl_ctx* c, unsigned* start) {
    // hook: 1: goals that need arrivals that never come; 2: the first barriers wrap
    const int test = c->barrier_test;
    c->barrier_test = 0;
    const unsigned near_wrap = 0xffffffc0u;
    *start = test == 1 ? 0x40000000u : test == 2 ? near_wrap : 0u;
    return test == 2 ? cudaMemcpyAsync(c->dbar.p, &near_wrap, sizeof(unsigned), cudaMemcpyHostToDevice, c->stream)
                     : cudaMemsetAsync(c->dbar.p, 0, sizeof(unsigned), c->stream);
}

static int read_scal(isl_ctx* c) {
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->hscal, c->dscal.p, sizeof(CGScal), cudaMemcpyDeviceToHost, c->stream));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    return ISL_OK;
}

static int ensure_work(isl_ctx* c) {
    const size_t n = (size_t)c->neq;
    // FP32 vectors of the block solver live in the (padded) block space
    const size_t n32 = std::max(n, c->blocked ? (size_t)(3 * c->nbr) : (size_t)0);
    if (c->w64.n < 6 * n) ISL_CHECK_CUDA(c, c->w64.alloc(6 * n));
    if (c->w32.n < 6 * n32) ISL_CHECK_CUDA(c, c->w32.alloc(6 * n32));
    // partial sums: two per block of every grid used (at most 16 blocks per SM)
    const size_t maxgrid = (size_t)16 * c->sm_count;
    if (c->dpart.n < 2 * maxgrid + 64) ISL_CHECK_CUDA(c, c->dpart.alloc(2 * maxgrid + 64));
    if (!c->dscal.p) ISL_CHECK_CUDA(c, c->dscal.alloc(2));
    if (!c->dbar.p) {
        ISL_CHECK_CUDA(c, c->dbar.alloc(2));
        ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dbar.p, 0, 2 * sizeof(unsigned), c->stream));
    }
    return ISL_OK;
}

// plain FP64 CG
static int solve_fp64(isl_ctx* c, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* nc) {
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq;
    double* W = c->w64.p;
    double *x = W, *r = W + n, *p = W + 2 * n, *q = W + 3 * n, *dinv = W + 4 * n;
    if (!c->spmv_lpr64) c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, c->drhs.p, q, c->dscal.p, c->dpart.p);
    const int mi = (int)std::min<int64_t>(max_iter, INT32_MAX - 1);
    const unsigned grid = vec_grid(c);
    k_dinv<double, double><<<grid, BS, 0, st>>>((int)n, c->ddiag.p, c->dval64.p, dinv);
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dscal.p, 0, sizeof(CGScal), st));
    k_cg_init<double, double><<<grid, BS, 0, st>>>((int)n, c->drhs.p, x, r, p, dinv, c->dscal.p, c->dpart.p, tol, 0.0);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 2;
    cudaGraphExec_t exec;
    int rc = capture_chunk<double, double>(c, c->dval64.p, x, r, p, q, dinv, c->spmv_lpr64, mi, &exec);
    if (rc != ISL_OK) return rc;
    const int64_t max_replays = (int64_t)mi / CHUNK + 3;
    int64_t replays = 0;
    for (;;) {
        rc = read_scal(c);
        if (rc != ISL_OK) break;
        if (c->hscal->done) break;
        if (++replays > max_replays) { rc = ISL_ERR_TIMEOUT; c->err = "CG made no progress"; break; }
        if (cudaGraphLaunch(exec, st) != cudaSuccess) { rc = ISL_ERR_CUDA; c->err = "graph launch failed"; break; }
        c->launches += 3 * CHUNK;
    }
    cudaGraphExecDestroy(exec);
    if (rc != ISL_OK) return rc;
    const CGScal& h = *c->hscal;
    if (h.bad) ISL_FAIL(c, ISL_ERR_NAN, "CG breakdown (non-finite reduction)");
    *iters = h.iters;
    *rel = h.rhsNorm2 > 0 ? std::sqrt(h.rr / h.rhsNorm2) : 0.0;
    *nc = (h.done == 2);
    k_copy64<<<grid, BS, 0, st>>>((int)n, x, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}

// FP32 CG with FP64 reliable updates
// ---------------------------------------------------------------------------
// Small scalar systems: the whole mixed solve in one thread-block cluster.
// The CTAs of one cluster split the rows; hardware cluster barriers separate
// the phases and the partial sums are exchanged through distributed shared
// memory, every CTA adding the CTAs' sums in rank order (so all CTAs hold the
// same scalars).  The FP32 iterations and the FP64 reliable updates (fold,
// b - A64 x, restart) all run inside the one launch, with the recurrences of
// the graph path (k_cg_dir, k_spmv_pap, k_cg_update, k_fold, k_residual64,
// k_restart32).
namespace cgrp = cooperative_groups;
constexpr int CL_BS = 1024;
constexpr int CLUSTER_MAX_N = 65536;

// row . v with plain (coherent) loads of v: v is written inside the launch
template <typename TV, typename TX, int LPR>
__device__ inline TX row_dot_c(int row, bool active, const int* __restrict__ rowptr, const int* __restrict__ colind,
                               const TV* __restrict__ val, const TX* v, int lane) {
    TX acc = TX(0);
    if (active) {
        const int lo = __ldg(rowptr + row), hi = __ldg(rowptr + row + 1);
        for (int k = lo + lane; k < hi; k += LPR) acc += (TX)__ldg(val + k) * v[__ldg(colind + k)];
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, LPR);
    return acc;
}

// sums of (a, b) over all threads of the cluster, in a fixed order: each CTA
// reduces its threads (one pass for both values; the warps in the values'
// precision, the warp sums in FP64 by one warp), lane k of warp 0 reads CTA
// k's pair through distributed shared memory, and a fixed shuffle tree adds
// the CTAs (so every CTA holds the same totals).  The slot cycles, so a CTA
// never rewrites a slot that a peer may still read.
template <typename T>
__device__ inline void cluster_sum2(T a, T b, double (*red)[2], int& slot, double* sh, double* bc, double& ta, double& tb) {
    cgrp::cluster_group cl = cgrp::this_cluster();
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) {  // within a warp in the values' own precision
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    __syncthreads();  // sh is free (previous users are done)
    if (l == 0) { sh[2 * w] = (double)a; sh[2 * w + 1] = (double)b; }
    __syncthreads();
    if (w == 0) {
        const int nw = (int)(blockDim.x >> 5);
        double u = l < nw ? sh[2 * l] : 0.0, v = l < nw ? sh[2 * l + 1] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            u += __shfl_xor_sync(0xffffffffu, u, o);
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (l == 0) { red[slot][0] = u; red[slot][1] = v; }
    }
    cl.sync();
    if (w == 0) {
        const int n = (int)cl.num_blocks();
        double u = 0.0, v = 0.0;
        if (l < n) {
            const double* peer = cl.map_shared_rank(&red[slot][0], l);
            u = peer[0];
            v = peer[1];
        }
        for (int o = 16; o > 0; o >>= 1) {
            u += __shfl_xor_sync(0xffffffffu, u, o);
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (l == 0) { bc[0] = u; bc[1] = v; }
    }
    __syncthreads();
    ta = bc[0];
    tb = bc[1];
    slot = (slot + 1) & 3;
}

// Scalar state of the one-cluster CG.  Thread 0 of each CTA holds it (every
// CTA computes the same values from the same sums); the other threads get
// alpha and beta in FP32 and a control code through shared memory, so the
// FP64 divisions and tests run once per CTA instead of once per thread.
struct ClusterScalars {
    double rz, rz_old, beta, rr, thr, trig, rr_true;
    int iters, max_iter, exact64, bad, nupd;
};
enum { CTL_GO = 0, CTL_DONE = 1, CTL_MAX = 2, CTL_UPDATE = 3, CTL_BAD = 4 };

__device__ inline float cs_alpha(ClusterScalars& s, double pap, float* sf) {
    if (threadIdx.x == 0) sf[0] = (float)(s.rz / pap);
    __syncthreads();
    return sf[0];  // rewritten only after later barriers
}

// after the (r.r, r.z) sums of an iteration; beta for the next direction in sf[1]
__device__ inline int cs_update(ClusterScalars& s, double trr, double trz, float* sf, int* si) {
    if (threadIdx.x == 0) {
        s.iters += 1;
        s.rr = trr;
        s.rz_old = s.rz;
        s.beta = trz / s.rz;
        s.rz = trz;
        int ctl = CTL_GO;
        if (!(trr == trr) || !(trz == trz)) { s.bad = 1; ctl = CTL_BAD; }
        else if (!s.exact64) {
            // FP32 CG on the iterated residual (inexact Newton steps)
            if (trr < s.thr) ctl = CTL_DONE;
            else if (s.iters >= s.max_iter) ctl = CTL_MAX;
            if (ctl != CTL_GO) s.rr_true = trr;
        } else if (trr < s.thr || trr < s.trig || s.iters >= s.max_iter) {
            ctl = CTL_UPDATE;
        }
        sf[1] = (float)s.beta;
        si[0] = ctl;
    }
    __syncthreads();
    return si[0];
}

// after the FP64 residual of a reliable update: converged, iteration limit,
// breakdown, or a restart from the true residual with the same direction
// (fresh directions, beta = 0, when the true residual has not dropped since
// the previous reliable update: the FP32 directions have lost conjugacy)
__device__ inline int cs_residual(ClusterScalars& s, double rr_true, double rr_restart, double rz_restart, float* sf, int* si) {
    if (threadIdx.x == 0) {
        const bool fresh = s.nupd > 0 && rr_true >= s.rr_true;
        s.rr_true = rr_true;
        s.nupd += 1;
        int ctl = CTL_GO;
        if (!(rr_true == rr_true)) { s.bad = 1; ctl = CTL_BAD; }
        else if (rr_true <= s.thr) ctl = CTL_DONE;
        else if (s.iters >= s.max_iter) ctl = CTL_MAX;
        else {
            s.rr = rr_restart;
            s.beta = fresh ? 0.0 : rz_restart / s.rz_old;
            s.rz = rz_restart;
            s.trig = kDelta2 * rr_true;
            sf[1] = (float)s.beta;
        }
        si[0] = ctl;
    }
    __syncthreads();
    return si[0];
}

__device__ inline ClusterScalars cs_load(const CGScal* S, int max_iter, int exact64) {
    ClusterScalars s;
    s.rz = S->absNew;
    s.rz_old = S->absOld;
    s.beta = S->beta;
    s.rr = S->rr;
    s.thr = S->threshold;
    s.trig = S->rrtrig;
    s.rr_true = S->rhsNorm2;
    s.iters = S->iters;
    s.max_iter = max_iter;
    s.exact64 = exact64;
    s.bad = 0;
    s.nupd = 0;
    return s;
}

__device__ inline void cs_store(const ClusterScalars& s, int done, CGScal* S) {
    S->rr = s.rr;
    S->rz = s.rr_true;
    S->iters = s.iters;
    S->absOld = s.rz_old;
    S->absNew = s.rz;
    S->beta = s.beta;
    if (s.bad) S->bad = 1;
    S->done = done;
}

template <int LPR>
__global__ void __launch_bounds__(CL_BS, 1) k_cg_cluster(int n, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                                         const float* __restrict__ val32, const double* __restrict__ val64,
                                                         const double* __restrict__ b, const float* __restrict__ dinv,
                                                         float* x32, float* r32, float* p32, float* q32, double* x64,
                                                         double* r64, CGScal* S, int max_iter, int exact64) {
    cgrp::cluster_group cl = cgrp::this_cluster();
    __shared__ double sh[2 * (CL_BS / 32)];
    __shared__ double red[4][2];
    __shared__ double bc[2];
    const int rank = (int)cl.block_rank(), ncta = (int)cl.num_blocks();
    const int r0 = (int)((long long)n * rank / ncta), r1 = (int)((long long)n * (rank + 1) / ncta);
    const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR, ngrp = CL_BS / LPR;
    const int wgrp = grp - grp % (32 / LPR);  // first row group of this warp: row loops stay warp-uniform
    int slot = 0;
    __shared__ float sf[2];
    __shared__ int si[1];
    ClusterScalars sc = cs_load(S, max_iter, exact64);
    int done = S->done;
    if (threadIdx.x == 0) sf[1] = (float)sc.beta;
    __syncthreads();
    double t0, t1;
    while (!done) {
        // p = D^-1 r + beta p
        const float fb = sf[1];
        for (int i = r0 + (int)threadIdx.x; i < r1; i += CL_BS) p32[i] = dinv[i] * r32[i] + fb * p32[i];
        cl.sync();
        // q = A p, p.q
        float loc = 0.f;
        for (int base = r0 + wgrp; base < r1; base += ngrp) {
            const int row = base + (grp - wgrp);
            const bool act = row < r1;
            const float acc = row_dot_c<float, float, LPR>(row, act, rowptr, colind, val32, p32, lane);
            if (act && lane == 0) {
                q32[row] = acc;
                loc += p32[row] * acc;
            }
        }
        cluster_sum2(loc, 0.f, red, slot, sh, bc, t0, t1);
        const float alpha = cs_alpha(sc, t0, sf);
        // x += alpha p, r -= alpha q; r.r, r.z
        float frr = 0.f, frz = 0.f;
        for (int i = r0 + (int)threadIdx.x; i < r1; i += CL_BS) {
            x32[i] += alpha * p32[i];
            const float ri = r32[i] - alpha * q32[i];
            r32[i] = ri;
            frr += ri * ri;
            frz += ri * (dinv[i] * ri);
        }
        cluster_sum2(frr, frz, red, slot, sh, bc, t0, t1);
        const int ctl = cs_update(sc, t0, t1, sf, si);
        if (ctl == CTL_BAD) { done = 1; break; }
        if (!exact64) {
            if (ctl != CTL_GO) {
                for (int i = r0 + (int)threadIdx.x; i < r1; i += CL_BS) { x64[i] += (double)x32[i]; x32[i] = 0.f; }
                done = ctl;
            }
            continue;
        }
        if (ctl == CTL_UPDATE) {
            // reliable update: fold the FP32 increment, true residual in FP64
            for (int i = r0 + (int)threadIdx.x; i < r1; i += CL_BS) { x64[i] += (double)x32[i]; x32[i] = 0.f; }
            cl.sync();
            double lt = 0.0, lrr = 0.0, lrz = 0.0;
            for (int base = r0 + wgrp; base < r1; base += ngrp) {
                const int row = base + (grp - wgrp);
                const bool act = row < r1;
                const double ax = row_dot_c<double, double, LPR>(row, act, rowptr, colind, val64, x64, lane);
                if (act && lane == 0) {
                    const double ri = b[row] - ax;
                    r64[row] = ri;
                    lt += ri * ri;
                    // the restart residual (FP32) and its sums, from the same pass
                    const float rf = (float)ri;
                    r32[row] = rf;
                    lrr += (double)rf * (double)rf;
                    lrz += (double)rf * (double)(dinv[row] * rf);
                }
            }
            cluster_sum2(lt, lrr, red, slot, sh, bc, t0, t1);
            const double rr_true = t0, rr_restart = t1;
            cluster_sum2(lrz, 0.0, red, slot, sh, bc, t0, t1);
            const int c2 = cs_residual(sc, rr_true, rr_restart, t0, sf, si);
            if (c2 != CTL_GO) { done = c2 == CTL_MAX ? 2 : 1; break; }
        }
    }
    if (rank == 0 && threadIdx.x == 0) cs_store(sc, done, S);
    // no CTA may leave while a peer can still read its shared memory
    cl.sync();
}

// The same solve with the cluster's rows kept on chip: each CTA copies its
// slice of the FP32 CSR matrix and of x, r, p, q and D^-1 into shared memory
// once; the SpMV reads the p entries of other CTAs through distributed shared
// memory (owner rank = column / chunk).  Only the FP64 reliable updates read
// the FP64 matrix and the FP64 iterate from global memory.  Used when a CTA's
// slice fits in shared memory.
template <int LPR>
__global__ void __launch_bounds__(CL_BS, 1) k_cg_cluster_smem(int n, int chunk, const int* __restrict__ rowptr,
                                                              const int* __restrict__ colind, const float* __restrict__ val32,
                                                              const double* __restrict__ val64, const double* __restrict__ b,
                                                              const float* __restrict__ dinvg, double* x64, CGScal* S,
                                                              int max_iter, int exact64, int max_nnz) {
    cgrp::cluster_group cl = cgrp::this_cluster();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double sh[2 * (CL_BS / 32)];
    __shared__ double red[4][2];
    __shared__ double bc[2];
    const int rank = (int)cl.block_rank();
    const int r0 = min(n, rank * chunk), r1 = min(n, r0 + chunk), nloc = r1 - r0;
    int* rp = (int*)smem;                // [chunk + 1]
    int* cs = rp + (chunk + 1);          // [max_nnz]
    float* vs = (float*)(cs + max_nnz);  // [max_nnz]
    float* xs = vs + max_nnz;            // [chunk] each: x, r, p, q, D^-1
    float* rs = xs + chunk;
    float* ps = rs + chunk;
    float* qs = ps + chunk;
    float* ds = qs + chunk;
    const int base = rowptr[r0];
    const int nnzl = rowptr[r1] - base;
    for (int i = (int)threadIdx.x; i <= nloc; i += CL_BS) rp[i] = rowptr[r0 + i] - base;
    for (int k = (int)threadIdx.x; k < nnzl; k += CL_BS) { cs[k] = colind[base + k]; vs[k] = val32[base + k]; }
    for (int i = (int)threadIdx.x; i < nloc; i += CL_BS) {
        xs[i] = 0.f;
        rs[i] = (float)b[r0 + i];
        ps[i] = 0.f;
        ds[i] = dinvg[r0 + i];
    }
    const int lane = threadIdx.x % LPR, grp = threadIdx.x / LPR, ngrp = CL_BS / LPR;
    const int wgrp = grp - grp % (32 / LPR);  // row loops stay warp-uniform
    int slot = 0;
    __shared__ float sf[2];
    __shared__ int si[1];
    ClusterScalars sc = cs_load(S, max_iter, exact64);
    int done = S->done;
    if (threadIdx.x == 0) sf[1] = (float)sc.beta;
    double t0, t1;
    cl.sync();
    while (!done) {
        // p = D^-1 r + beta p
        const float fb = sf[1];
        for (int i = (int)threadIdx.x; i < nloc; i += CL_BS) ps[i] = ds[i] * rs[i] + fb * ps[i];
        cl.sync();
        // q = A p (p of other CTAs through distributed shared memory), p.q
        float loc = 0.f;
        for (int bi = wgrp; bi < nloc; bi += ngrp) {
            const int row = bi + (grp - wgrp);
            const bool act = row < nloc;
            float acc = 0.f;
            if (act)
                for (int k = rp[row] + lane; k < rp[row + 1]; k += LPR) {
                    const int c = cs[k], owner = c / chunk, li = c - owner * chunk;
                    const float pv = owner == rank ? ps[li] : *cl.map_shared_rank(ps + li, owner);
                    acc += vs[k] * pv;
                }
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, LPR);
            if (act && lane == 0) {
                qs[row] = acc;
                loc += ps[row] * acc;
            }
        }
        cluster_sum2(loc, 0.f, red, slot, sh, bc, t0, t1);
        const float alpha = cs_alpha(sc, t0, sf);
        // x += alpha p, r -= alpha q; r.r, r.z
        float frr = 0.f, frz = 0.f;
        for (int i = (int)threadIdx.x; i < nloc; i += CL_BS) {
            xs[i] += alpha * ps[i];
            const float ri = rs[i] - alpha * qs[i];
            rs[i] = ri;
            frr += ri * ri;
            frz += ri * (ds[i] * ri);
        }
        cluster_sum2(frr, frz, red, slot, sh, bc, t0, t1);
        const int ctl = cs_update(sc, t0, t1, sf, si);
        if (ctl == CTL_BAD) { done = 1; break; }
        if (!exact64) {
            if (ctl != CTL_GO) {
                for (int i = (int)threadIdx.x; i < nloc; i += CL_BS) { x64[r0 + i] += (double)xs[i]; xs[i] = 0.f; }
                done = ctl;
            }
            continue;
        }
        if (ctl == CTL_UPDATE) {
            // reliable update: fold, true residual in FP64 from global memory;
            // the rounded residual and its sums for a restart come from the same pass
            for (int i = (int)threadIdx.x; i < nloc; i += CL_BS) { x64[r0 + i] += (double)xs[i]; xs[i] = 0.f; }
            cl.sync();
            double lt = 0.0, lrr = 0.0, lrz = 0.0;
            for (int bi = wgrp; bi < nloc; bi += ngrp) {
                const int row = bi + (grp - wgrp);
                const bool act = row < nloc;
                const double ax = row_dot_c<double, double, LPR>(r0 + row, act, rowptr, colind, val64, x64, lane);
                if (act && lane == 0) {
                    const double ri = b[r0 + row] - ax;
                    lt += ri * ri;
                    const float rf = (float)ri;
                    rs[row] = rf;
                    lrr += (double)rf * (double)rf;
                    lrz += (double)rf * (double)(ds[row] * rf);
                }
            }
            cluster_sum2(lt, lrr, red, slot, sh, bc, t0, t1);
            const double rr_true = t0, rr_restart = t1;
            cluster_sum2(lrz, 0.0, red, slot, sh, bc, t0, t1);
            const int c2 = cs_residual(sc, rr_true, rr_restart, t0, sf, si);
            if (c2 != CTL_GO) { done = c2 == CTL_MAX ? 2 : 1; break; }
        }
    }
    if (rank == 0 && threadIdx.x == 0) cs_store(sc, done, S);
    // no CTA may leave while a peer can still read its shared memory
    cl.sync();
}

template <int LPR>
static cudaError_t launch_cluster_smem(int ncta, size_t smem, cudaStream_t st, int n, int chunk, const int* rp, const int* ci,
                                       const float* v32, const double* v64, const double* b, const float* dinv, double* x64,
                                       CGScal* S, int mi, int exact64, int max_nnz) {
    cudaError_t e = cudaFuncSetAttribute(k_cg_cluster_smem<LPR>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cg_cluster_smem<LPR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(CL_BS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ncta;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int nclusters = 0;
    e = cudaOccupancyMaxActiveClusters(&nclusters, k_cg_cluster_smem<LPR>, &cfg);
    if (e != cudaSuccess) return e;
    if (nclusters < 1) return cudaErrorInvalidConfiguration;
    return cudaLaunchKernelEx(&cfg, k_cg_cluster_smem<LPR>, n, chunk, rp, ci, v32, v64, b, dinv, x64, S, mi, exact64, max_nnz);
}

template <int LPR>
static cudaError_t launch_cluster(int ncta, cudaStream_t st, int n, const int* rp, const int* ci, const float* v32,
                                  const double* v64, const double* b, const float* dinv, float* x32, float* r32, float* p32,
                                  float* q32, double* x64, double* r64, CGScal* S, int mi, int exact64) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(CL_BS);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ncta;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_cg_cluster<LPR>, n, rp, ci, v32, v64, b, dinv, x32, r32, p32, q32, x64, r64, S, mi,
                              exact64);
}

// CTAs of the cluster: 16 where the device allows that size, else 8; 0 when
// cluster launches are unavailable
template <int LPR>
static int probe_cluster(isl_ctx* c) {
    int ok = 0;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrClusterLaunch, c->device) != cudaSuccess || !ok) return 0;
    cudaFuncSetAttribute(k_cg_cluster<LPR>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int ncta : {16, 8}) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ncta);
        cfg.blockDim = dim3(CL_BS);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = ncta;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, k_cg_cluster<LPR>, &cfg) == cudaSuccess && nclusters > 0) return ncta;
    }
    cudaGetLastError();
    return 0;
}

int cluster_ctas(isl_ctx* c) {
    if (c->cluster_size < 0) {
        // every LPR variant shares the size limits; probe all so that each can be launched
        int a = probe_cluster<2>(c), b = probe_cluster<4>(c), d = probe_cluster<8>(c), e = probe_cluster<16>(c),
            f = probe_cluster<32>(c);
        c->cluster_size = std::min(std::min(std::min(a, b), std::min(d, e)), f);
        cudaGetLastError();
    }
    return c->cluster_size;
}

static int solve_mixed_cluster(isl_ctx* c, int ncta, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* nc) {
    cudaStream_t st = c->stream;
    const int n = (int)c->neq;
    double* W = c->w64.p;
    double *x64 = W, *r64 = W + n;
    float* V = c->w32.p;
    float *x32 = V, *r32 = V + n, *p32 = V + 2 * n, *q32 = V + 3 * n, *d32 = V + 4 * n;
    const int mi = (int)std::min<int64_t>(max_iter, INT32_MAX - 1);
    const unsigned grid = vec_grid(c);
    CGScal* S = c->dscal.p;
    const int exact64 = c->have64 ? 1 : 0;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dscal.p, 0, sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(x64, 0, (size_t)n * 8, st));
    k_dinv<float, float><<<grid, BS, 0, st>>>(n, c->ddiag.p, c->dval32.p, d32);
    k_cg_init<double, float><<<grid, BS, 0, st>>>(n, c->drhs.p, x32, r32, p32, d32, S, c->dpart.p, tol, exact64 ? kDelta2 : 0.0);
    // lanes per row: from the mean row length, but few enough that the rows of
    // one CTA take a single pass of its threads
    const double avg = (double)c->nnz / (double)n;
    int lpr = 2;
    while (lpr < 32 && lpr < avg / 2) lpr *= 2;
    const int rows_per_cta = (n + ncta - 1) / ncta;
    while (lpr > 2 && (long long)rows_per_cta * lpr > CL_BS) lpr /= 2;
    cudaError_t e = cudaErrorInvalidConfiguration;
    // on-chip variant when each CTA's slice fits in shared memory
    size_t smem = 0;
    int max_nnz = 0;
    const int chunk = rows_per_cta;
    if ((int64_t)c->hrp_small.size() == (int64_t)n + 1) {
        for (int r = 0; r < ncta; ++r) {
            const int a0 = std::min(n, r * chunk), a1 = std::min(n, a0 + chunk);
            max_nnz = std::max(max_nnz, c->hrp_small[a1] - c->hrp_small[a0]);
        }
        smem = (size_t)4 * (chunk + 1) + (size_t)8 * max_nnz + (size_t)20 * chunk;
    }
    const bool onchip = smem > 0 && smem <= (size_t)200 * 1024;
    if (onchip) {
        switch (lpr) {
            case 2: e = launch_cluster_smem<2>(ncta, smem, st, n, chunk, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x64, S, mi, exact64, max_nnz); break;
            case 4: e = launch_cluster_smem<4>(ncta, smem, st, n, chunk, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x64, S, mi, exact64, max_nnz); break;
            case 8: e = launch_cluster_smem<8>(ncta, smem, st, n, chunk, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x64, S, mi, exact64, max_nnz); break;
            case 16: e = launch_cluster_smem<16>(ncta, smem, st, n, chunk, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x64, S, mi, exact64, max_nnz); break;
            default: e = launch_cluster_smem<32>(ncta, smem, st, n, chunk, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x64, S, mi, exact64, max_nnz); break;
        }
        if (e != cudaSuccess) cudaGetLastError();  // not launchable here: the global-memory variant runs
    }
    if (e != cudaSuccess)
    switch (lpr) {
        case 2: e = launch_cluster<2>(ncta, st, n, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x32, r32, p32, q32, x64, r64, S, mi, exact64); break;
        case 4: e = launch_cluster<4>(ncta, st, n, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x32, r32, p32, q32, x64, r64, S, mi, exact64); break;
        case 8: e = launch_cluster<8>(ncta, st, n, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x32, r32, p32, q32, x64, r64, S, mi, exact64); break;
        case 16: e = launch_cluster<16>(ncta, st, n, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x32, r32, p32, q32, x64, r64, S, mi, exact64); break;
        default: e = launch_cluster<32>(ncta, st, n, c->drowptr.p, c->dcolind.p, c->dval32.p, c->dval64.p, c->drhs.p, d32, x32, r32, p32, q32, x64, r64, S, mi, exact64); break;
    }
    ISL_CHECK_CUDA(c, e);
    c->launches += 3;
    int rc = read_scal(c);
    if (rc != ISL_OK) return rc;
    const CGScal& h = *c->hscal;
    if (h.bad) ISL_FAIL(c, ISL_ERR_NAN, "CG breakdown (non-finite reduction)");
    const double bnorm2 = h.rhsNorm2;
    *iters = h.iters;
    *rel = bnorm2 > 0 ? std::sqrt((h.iters > 0 ? h.rz : bnorm2) / bnorm2) : 0.0;
    *nc = (h.done == 2);
    k_copy64<<<grid, BS, 0, st>>>(n, x64, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}

static int solve_mixed(isl_ctx* c, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* nc) {
    if (c->use_persist != 0 && c->neq <= CLUSTER_MAX_N) {
        const int ncta = cluster_ctas(c);
        if (ncta > 0) return solve_mixed_cluster(c, ncta, tol, max_iter, iters, rel, nc);
    }
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq;
    double* W = c->w64.p;
    double *x64 = W, *r64 = W + n;
    float* V = c->w32.p;
    float *x32 = V, *r32 = V + n, *p32 = V + 2 * n, *q32 = V + 3 * n, *d32 = V + 4 * n;
    int rc = ensure_ssell(c);
    if (rc != ISL_OK) return rc;
    if (!c->spmv_lpr32) {
        ISL_CHECK_CUDA(c, cudaMemsetAsync(p32, 0, n * 4, st));
        c->spmv_lpr32 = autotune_spmv32(c, p32, q32, c->dscal.p, c->dpart.p);
    }
    c->spmv32_used = c->spmv_lpr32;
    const bool exact64 = c->have64;  // without the FP64 matrix: plain FP32 CG (inexact Newton tangents)
    if (exact64 && !c->spmv_lpr64)
        c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, c->drhs.p, W + 3 * n, c->dscal.p, c->dpart.p);
    const int mi = (int)std::min<int64_t>(max_iter, INT32_MAX - 1);
    const unsigned grid = vec_grid(c);
    CGScal* S = c->dscal.p;
    double* dres = (double*)(c->dscal.p + 1);
    unsigned* ticket = &(c->dscal.p + 1)->ticket1;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dscal.p, 0, 2 * sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(x64, 0, n * 8, st));
    k_dinv<float, float><<<grid, BS, 0, st>>>((int)n, c->ddiag.p, c->dval32.p, d32);
    k_cg_init<double, float><<<grid, BS, 0, st>>>((int)n, c->drhs.p, x32, r32, p32, d32, S, c->dpart.p, tol,
                                                   c->have64 ? c->ru_drop2 : 0.0);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 2;
    cudaGraphExec_t exec;
    rc = capture_chunk<float, float>(c, c->dval32.p, x32, r32, p32, q32, d32, c->spmv_lpr32, mi, &exec);
    if (rc != ISL_OK) return rc;
    rc = read_scal(c);
    const double bnorm2 = c->hscal->rhsNorm2;
    double rr_true = bnorm2;
    double rr_last = 0.0;  // true residual of the previous reliable update
    const int64_t max_replays = (int64_t)mi + 64;
    int64_t replays = 0;
    bool converged = (bnorm2 == 0.0);
    while (rc == ISL_OK && !converged) {
        if (++replays > max_replays) { rc = ISL_ERR_TIMEOUT; c->err = "mixed CG made no progress"; break; }
        if (cudaGraphLaunch(exec, st) != cudaSuccess) { rc = ISL_ERR_CUDA; c->err = "graph launch failed"; break; }
        c->launches += 3 * CHUNK;
        rc = read_scal(c);
        if (rc != ISL_OK) break;
        const CGScal h = *c->hscal;
        if (h.bad) { rc = ISL_ERR_NAN; c->err = "CG breakdown (non-finite reduction)"; break; }
        const bool at_max = h.iters >= mi;
        if (!exact64) {
            if (h.done || at_max) {
                k_fold<<<grid, BS, 0, st>>>((int)n, x32, x64);
                c->launches += 1;
                rr_true = h.rr;
                converged = h.done == 1;
                if (!converged) *nc = true;
                break;
            }
            continue;
        }
        if (h.done || at_max) {
            // reliable update: true residual in FP64
            k_fold<<<grid, BS, 0, st>>>((int)n, x32, x64);
            launch_residual(c->spmv_lpr64, grid, st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, x64, c->drhs.p, r64,
                            c->dpart.p, ticket, dres);
            c->launches += 2;
            ISL_CHECK_CUDA(c, cudaMemcpyAsync(&rr_true, dres, 8, cudaMemcpyDeviceToHost, st));
            ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
            if (!(rr_true == rr_true)) { rc = ISL_ERR_NAN; c->err = "refinement residual is not finite"; break; }
            if (rr_true <= tol * tol * bnorm2) { converged = true; break; }
            if (at_max) { *nc = true; break; }
            const int fresh = (rr_last > 0.0 && rr_true >= rr_last) ? 1 : 0;
            rr_last = rr_true;
            k_restart32<<<grid, BS, 0, st>>>((int)n, r64, r32, d32, S, c->dpart.p, c->ru_drop2 * rr_true, fresh);
            c->launches += 1;
        }
    }
    cudaGraphExecDestroy(exec);
    if (rc != ISL_OK) return rc;
    if (!converged && bnorm2 > 0) *nc = true;
    rc = read_scal(c);
    if (rc != ISL_OK) return rc;
    *iters = c->hscal->iters;
    *rel = bnorm2 > 0 ? std::sqrt(rr_true / bnorm2) : 0.0;
    k_copy64<<<grid, BS, 0, st>>>((int)n, x64, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}


// ===========================================================================
// Node-blocked (3x3 BSR) FP32 path of the mixed solver.  Every DOF object of
// a 3-component field with all components active gives three consecutive
// equations, so the CSR pattern is the node graph times 3x3 blocks.  The
// block copy stores 4 bytes of column index per 9 values (4.4 bytes per
// nonzero instead of 8), and the preconditioner inverts the 3x3 diagonal
// blocks (block Jacobi).
__global__ void k_bsr_pattern(int nbr, const int* __restrict__ rowptr, const int* __restrict__ colind, int* __restrict__ bptr,
                              int* __restrict__ bcol, int* __restrict__ brow, int* __restrict__ bad) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbr; i += gridDim.x * blockDim.x) {
        const int r0 = rowptr[3 * i], len = rowptr[3 * i + 1] - r0;
        const int b0 = r0 / 9;
        bptr[i] = b0;
        if (i == nbr - 1) bptr[nbr] = rowptr[3 * nbr] / 9;
        if (r0 % 9 != 0 || len % 3 != 0 || rowptr[3 * i + 2] - rowptr[3 * i + 1] != len ||
            rowptr[3 * i + 3] - rowptr[3 * i + 2] != len) {
            atomicOr(bad, 1);
            continue;
        }
        for (int k = 0; k < len / 3; ++k) {
            const int j3 = colind[r0 + 3 * k];
            if (j3 % 3 != 0) atomicOr(bad, 1);
            for (int r = 0; r < 3; ++r)
                for (int cc = 0; cc < 3; ++cc)
                    if (colind[rowptr[3 * i + r] + 3 * k + cc] != j3 + cc) atomicOr(bad, 1);
            bcol[b0 + k] = j3 / 3;
            brow[b0 + k] = i;
        }
    }
}

__global__ void k_bsr_values(int nblk, const int* __restrict__ brow, const int* __restrict__ bptr, const int* __restrict__ rowptr,
                             const float* __restrict__ v32, const int* __restrict__ sdst, float* __restrict__ sv,
                             float* __restrict__ bv) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += gridDim.x * blockDim.x) {
        const int i = brow[b], k = b - bptr[i];
        const size_t slot = (size_t)sdst[b];
        const size_t g = slot >> 5, l = slot & 31;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int o = rowptr[3 * i + r] + 3 * k;
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
                const float v = v32[o + cc];
                sv[(g * 9 + r * 3 + cc) * 32 + l] = v;
                bv[(size_t)(r * 3 + cc) * nblk + b] = v;
            }
        }
    }
}

// 16-bit copy of the slot columns as offsets from the slot's block row; a
// padding row past nbr gets the offset of row nbr - 1 (a valid column), and
// any offset outside the 16-bit range sets *far
__global__ void k_sell_col16(int nbr, int nslice, const int* __restrict__ soff, const int* __restrict__ swid,
                             const int* __restrict__ scol, short* __restrict__ scol16, int* __restrict__ far) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nslice * 32; t += gridDim.x * blockDim.x) {
        const int s = t / 32, l = t % 32;
        const int o = soff[s], w = swid[s];
        const int i = s * 32 + l;
        for (int k = 0; k < w; ++k) {
            const int slot = o + k * 32 + l;
            const int off = i < nbr ? scol[slot] - i : (nbr - 1) - i;
            if (off < -32767 || off > 32767) { atomicOr(far, 1); scol16[slot] = 0; }
            else scol16[slot] = (short)off;
        }
    }
}

// Padded node blocks.  A DOF object with some of its three components
// constrained keeps a block row; aeq[3 I + c] is the equation of component c
// of block row I (-1: constrained).  The equations of a DOF object's active
// components are consecutive and increase with the object, so the lead row
// (first active component) of I lists, for every block column J, the run of
// J's equations eqf(J) .. eqf(J) + nact(J) - 1 in order.  Pass 0 counts the
// runs of every block row (and flags any row that is not of this form: a run
// that does not start at eqf(J), has the wrong length, or an active row of I
// whose columns differ from the lead row's); pass 1 writes the block columns,
// the block rows and the CSR position base of each block.
__device__ __forceinline__ int pad_first_eq(const int* __restrict__ aeq, int i) {
    const int e0 = aeq[3 * i], e1 = aeq[3 * i + 1], e2 = aeq[3 * i + 2];
    return e0 >= 0 ? e0 : (e1 >= 0 ? e1 : e2);
}
__device__ __forceinline__ int pad_nact(const int* __restrict__ aeq, int i) {
    return (aeq[3 * i] >= 0) + (aeq[3 * i + 1] >= 0) + (aeq[3 * i + 2] >= 0);
}
__global__ void k_bsr_pattern_pad(int nbr, int pass, const int* __restrict__ aeq, const int* __restrict__ eqblk,
                                  const int* __restrict__ rowptr, const int* __restrict__ colind, int* __restrict__ cnt,
                                  const int* __restrict__ bptr, int* __restrict__ bcol, int* __restrict__ brow,
                                  int* __restrict__ bcb, int* __restrict__ bad) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbr; i += gridDim.x * blockDim.x) {
        const int e0 = pad_first_eq(aeq, i);
        const int lo = rowptr[e0], len = rowptr[e0 + 1] - lo;
        int nb = 0, bad_i = 0;
        for (int k = 0; k < len;) {
            const int j = eqblk[colind[lo + k]];
            const int f = pad_first_eq(aeq, j), m = pad_nact(aeq, j);
            if (colind[lo + k] != f || k + m > len) { bad_i = 1; break; }
            for (int t = 1; t < m; ++t)
                if (colind[lo + k + t] != f + t) bad_i = 1;
            if (pass == 1) {
                const int b = bptr[i] + nb;
                bcol[b] = j;
                brow[b] = i;
                bcb[b] = k - f;
            }
            ++nb;
            k += m;
        }
        if (pass == 0) {
            for (int r = 0; r < 3 && !bad_i; ++r) {
                const int e = aeq[3 * i + r];
                if (e < 0 || e == e0) continue;
                if (rowptr[e + 1] - rowptr[e] != len) { bad_i = 1; break; }
                for (int k = 0; k < len; ++k)
                    if (colind[rowptr[e] + k] != colind[lo + k]) { bad_i = 1; break; }
            }
            cnt[i] = nb;
            if (bad_i) atomicOr(bad, 1);
        }
    }
}

// padded block values from the FP32 CSR values: constrained rows and columns
// hold zeros
__global__ void k_bsr_values_pad(int nblk, const int* __restrict__ brow, const int* __restrict__ bcol,
                                 const int* __restrict__ bcb, const int* __restrict__ aeq, const int* __restrict__ rowptr,
                                 const float* __restrict__ v32, const int* __restrict__ sdst, float* __restrict__ sv,
                                 float* __restrict__ bv) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nblk; b += gridDim.x * blockDim.x) {
        const int i = brow[b], j = bcol[b], cb = bcb[b];
        const size_t slot = (size_t)sdst[b];
        const size_t g = slot >> 5, l = slot & 31;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int er = aeq[3 * i + r];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
                const int ec = aeq[3 * j + cc];
                const float v = (er >= 0 && ec >= 0) ? v32[rowptr[er] + cb + ec] : 0.f;
                sv[(g * 9 + r * 3 + cc) * 32 + l] = v;
                bv[(size_t)(r * 3 + cc) * nblk + b] = v;
            }
        }
    }
}

// slice widths (longest block row of each slice of 32)
__global__ void k_sell_width(int nbr, int nslice, const int* __restrict__ bptr, int* __restrict__ swid) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nslice; s += gridDim.x * blockDim.x) {
        int w = 0;
        for (int l = 0; l < 32; ++l) {
            const int i = s * 32 + l;
            if (i < nbr) w = max(w, bptr[i + 1] - bptr[i]);
        }
        swid[s] = w;
    }
}

// column ids of every slot (padding slots point at a valid column and keep
// value 0) and the slot of every stored block
__global__ void k_sell_fill(int nbr, int nslice, const int* __restrict__ bptr, const int* __restrict__ bcol,
                            const int* __restrict__ soff, const int* __restrict__ swid, int* __restrict__ scol,
                            int* __restrict__ sdst) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nslice * 32; i += gridDim.x * blockDim.x) {
        const int s = i / 32, l = i % 32;
        const int w = swid[s], o = soff[s];
        const int len = (i < nbr) ? bptr[i + 1] - bptr[i] : 0;
        for (int k = 0; k < w; ++k) {
            const int slot = o + k * 32 + l;
            if (k < len) {
                scol[slot] = bcol[bptr[i] + k];
                sdst[bptr[i] + k] = slot;
            } else {
                scol[slot] = (i < nbr) ? i : 0;
            }
        }
    }
}

// inverse of a 3x3 block in FP64 (identity for a singular or non-finite block)
__device__ inline void bj_invert(const double A[3][3], float* __restrict__ out) {
    const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
    const double c01 = A[1][2] * A[2][0] - A[1][0] * A[2][2];
    const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
    const double det = A[0][0] * c00 + A[0][1] * c01 + A[0][2] * c02;
    double Bi[3][3];
    if (det != 0.0 && det == det) {
        const double id = 1.0 / det;
        Bi[0][0] = c00 * id; Bi[1][0] = c01 * id; Bi[2][0] = c02 * id;
        Bi[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * id;
        Bi[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * id;
        Bi[2][1] = (A[0][1] * A[2][0] - A[0][0] * A[2][1]) * id;
        Bi[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * id;
        Bi[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * id;
        Bi[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * id;
    } else {
        for (int r = 0; r < 3; ++r)
            for (int cc = 0; cc < 3; ++cc) Bi[r][cc] = (r == cc) ? 1.0 : 0.0;
    }
    for (int r = 0; r < 3; ++r)
        for (int cc = 0; cc < 3; ++cc) out[r * 3 + cc] = (float)Bi[r][cc];
}

// inverse of the 3x3 diagonal blocks, computed in FP64 from the FP64 values
// when they exist
template <typename TV>
__global__ void k_block_jacobi(int nbr, const int* __restrict__ rowptr, const int* __restrict__ diag, const TV* __restrict__ val,
                               float* __restrict__ binv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbr; i += gridDim.x * blockDim.x) {
        const int k = (diag[3 * i] - rowptr[3 * i]) / 3;
        double A[3][3];
        for (int r = 0; r < 3; ++r)
            for (int cc = 0; cc < 3; ++cc) A[r][cc] = (double)val[rowptr[3 * i + r] + 3 * k + cc];
        bj_invert(A, binv + (size_t)i * 9);
    }
}

// the same on padded blocks: the active components' sub-block, the identity
// on constrained components (whose residual entries stay zero)
template <typename TV>
__global__ void k_block_jacobi_pad(int nbr, const int* __restrict__ aeq, const int* __restrict__ diag,
                                   const TV* __restrict__ val, float* __restrict__ binv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nbr; i += gridDim.x * blockDim.x) {
        double A[3][3];
        for (int r = 0; r < 3; ++r) {
            const int er = aeq[3 * i + r];
            for (int cc = 0; cc < 3; ++cc) {
                const int ec = aeq[3 * i + cc];
                A[r][cc] = (er >= 0 && ec >= 0) ? (double)val[diag[er] + (ec - er)] : (r == cc ? 1.0 : 0.0);
            }
        }
        bj_invert(A, binv + (size_t)i * 9);
    }
}

// padded blocks, reliable update part 1: fold the FP32 increment (padded
// space) into the FP64 iterate (equations)
__global__ void k_fold_pad(int na, const int* __restrict__ aeq, float* __restrict__ x32, double* __restrict__ x64) {
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < na; a += gridDim.x * blockDim.x) {
        const int e = aeq[a];
        if (e >= 0) x64[e] += (double)x32[a];
        x32[a] = 0.0f;
    }
}

// q = A p on the sliced-ELL blocks, one warp per slice and one lane per block
// row (no shuffles: every lane owns its three outputs); partial p.q; last
// block: alpha
template <int LPB>
__global__ void __launch_bounds__(BS) k_bspmv_pap(int nbr, int nslice, const int* __restrict__ soff, const int* __restrict__ swid,
                                                  const int* __restrict__ scol, const float* __restrict__ sv, long long nslot,
                                                  const float* __restrict__ p, float* __restrict__ q, CGScal* S, double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * BS + threadIdx.x) >> 5, nwarps = gridDim.x * (BS / 32);
    float loc = 0.f;
    for (int s = warp; s < nslice; s += nwarps) {
        const int i = s * 32 + lane;
        const int o = soff[s], w = swid[s];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll LPB
        for (int k = 0; k < w; ++k) {
            const int slot = o + k * 32 + lane;
            const int j = __ldg(scol + slot);
            const float* v = sv + (size_t)(slot >> 5) * 288 + lane;  // group of 32 slots: [9][32]
            const float x0 = __ldg(p + 3 * j), x1 = __ldg(p + 3 * j + 1), x2 = __ldg(p + 3 * j + 2);
            a0 += __ldg(v) * x0 + __ldg(v + 32) * x1 + __ldg(v + 64) * x2;
            a1 += __ldg(v + 96) * x0 + __ldg(v + 128) * x1 + __ldg(v + 160) * x2;
            a2 += __ldg(v + 192) * x0 + __ldg(v + 224) * x1 + __ldg(v + 256) * x2;
        }
        if (i < nbr) {
            q[3 * i] = a0; q[3 * i + 1] = a1; q[3 * i + 2] = a2;
            loc += p[3 * i] * a0 + p[3 * i + 1] * a1 + p[3 * i + 2] * a2;
        }
    }
    const double bsum = block_sum_f(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bsum;
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

// Same product with the loads of U slots issued before any of them is used:
// U column indices and 9U values, then the 3U gathers of p, then the FMAs in
// slot order (bit-identical sums to the kernel above).  More bytes in flight
// per lane for the latency-bound stream; the values and column ids are read
// once per product and bypass L1.  COH: p is written inside the same kernel
// (persistent CG), so it is read with ordinary (coherent) loads instead of
// the non-coherent path.
template <int U, bool COH>
__device__ __forceinline__ float bspmv_slices(int nbr, int nslice, const int* __restrict__ soff,
                                               const int* __restrict__ swid, const int* __restrict__ scol,
                                               const float* __restrict__ sv, const float* p, float* q, int warp,
                                               int nwarps) {
    const int lane = threadIdx.x & 31;
    float loc = 0.f;
    for (int s = warp; s < nslice; s += nwarps) {
        const int i = s * 32 + lane;
        const int o = soff[s], w = swid[s];  // o: multiple of 32; w: warp-uniform
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        for (int k = 0; k < w; k += U) {
            int j[U];
            float v[U][9];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u < w) {
                    j[u] = ld_stream(scol + o + (k + u) * 32 + lane);
                    const float* vp = sv + (size_t)((o >> 5) + k + u) * 288 + lane;
#pragma unroll
                    for (int e = 0; e < 9; ++e) v[u][e] = ld_stream(vp + 32 * e);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u < w) {
                    const float* pj = p + 3 * j[u];
                    const float x0 = COH ? pj[0] : __ldg(pj), x1 = COH ? pj[1] : __ldg(pj + 1),
                                x2 = COH ? pj[2] : __ldg(pj + 2);
                    a0 += v[u][0] * x0 + v[u][1] * x1 + v[u][2] * x2;
                    a1 += v[u][3] * x0 + v[u][4] * x1 + v[u][5] * x2;
                    a2 += v[u][6] * x0 + v[u][7] * x1 + v[u][8] * x2;
                }
            }
        }
        if (i < nbr) {
            q[3 * i] = a0; q[3 * i + 1] = a1; q[3 * i + 2] = a2;
            const float* pi = p + 3 * i;
            const float p0 = pi[0], p1 = pi[1], p2 = pi[2];
            loc += p0 * a0 + p1 * a1 + p2 * a2;
        }
    }
    return loc;
}

template <int U, int MINB>
__global__ void __launch_bounds__(BS, MINB) k_bspmv_batch(int nbr, int nslice, const int* __restrict__ soff,
                                                          const int* __restrict__ swid, const int* __restrict__ scol,
                                                          const float* __restrict__ sv, const float* __restrict__ p,
                                                          float* __restrict__ q, CGScal* S, double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const int warp = (blockIdx.x * BS + threadIdx.x) >> 5, nwarps = gridDim.x * (BS / 32);
    const float loc = bspmv_slices<U, false>(nbr, nslice, soff, swid, scol, sv, p, q, warp, nwarps);
    const double bsum = block_sum_f(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bsum;
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

// The same product with the direction update folded in: the previous update
// kernel left z = B^-1 r, and every column block of p is formed where it is
// read, p_j = z_j + beta p_old_j (one fmaf per entry, so every reader and the
// owning row compute the same bits).  The owner of block row i writes p_i to
// the other buffer; p_old is never written during the product, so no block
// reads a value another block has already replaced.  Which of the two
// buffers holds p_old follows the parity of the iteration count, which the
// update kernel advances: the captured graph stays the same for every chunk,
// and a reliable-update restart (which keeps p) needs no copy.
// TC = short: the slots hold the column as a 16-bit offset from the slot's
// block row (every offset of the matrix within +-32,767; 2 B per block
// instead of 4)
template <int U, typename TC>
__device__ __forceinline__ float bspmv_slices_dir(int nbr, int nslice, const int* __restrict__ soff,
                                                   const int* __restrict__ swid, const TC* __restrict__ scol,
                                                   const float* __restrict__ sv, const float* __restrict__ z,
                                                   const float* __restrict__ pold, float beta, float* __restrict__ pnew,
                                                   float* __restrict__ q, int warp, int nwarps) {
    const int lane = threadIdx.x & 31;
    float loc = 0.f;
    for (int s = warp; s < nslice; s += nwarps) {
        const int i = s * 32 + lane;
        const int o = soff[s], w = swid[s];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        for (int k = 0; k < w; k += U) {
            int j[U];
            float v[U][9];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u < w) {
                    j[u] = ld_stream(scol + o + (k + u) * 32 + lane) + (sizeof(TC) == 2 ? i : 0);
                    const float* vp = sv + (size_t)((o >> 5) + k + u) * 288 + lane;
#pragma unroll
                    for (int e = 0; e < 9; ++e) v[u][e] = ld_stream(vp + 32 * e);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u < w) {
                    const size_t b = 3 * (size_t)j[u];
                    const float x0 = fmaf(beta, __ldg(pold + b), __ldg(z + b));
                    const float x1 = fmaf(beta, __ldg(pold + b + 1), __ldg(z + b + 1));
                    const float x2 = fmaf(beta, __ldg(pold + b + 2), __ldg(z + b + 2));
                    a0 += v[u][0] * x0 + v[u][1] * x1 + v[u][2] * x2;
                    a1 += v[u][3] * x0 + v[u][4] * x1 + v[u][5] * x2;
                    a2 += v[u][6] * x0 + v[u][7] * x1 + v[u][8] * x2;
                }
            }
        }
        if (i < nbr) {
            const size_t b = 3 * (size_t)i;
            const float p0 = fmaf(beta, __ldg(pold + b), __ldg(z + b));
            const float p1 = fmaf(beta, __ldg(pold + b + 1), __ldg(z + b + 1));
            const float p2 = fmaf(beta, __ldg(pold + b + 2), __ldg(z + b + 2));
            pnew[b] = p0; pnew[b + 1] = p1; pnew[b + 2] = p2;
            q[b] = a0; q[b + 1] = a1; q[b + 2] = a2;
            loc += p0 * a0 + p1 * a1 + p2 * a2;
        }
    }
    return loc;
}

template <int U, int MINB, typename TC>
__global__ void __launch_bounds__(BS, MINB) k_bspmv_dir(int nbr, int nslice, const int* __restrict__ soff,
                                                        const int* __restrict__ swid, const TC* __restrict__ scol,
                                                        const float* __restrict__ sv, const float* __restrict__ z,
                                                        float* pa, float* pb, float* __restrict__ q, CGScal* S,
                                                        double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const bool odd = S->iters & 1;
    const float beta = (float)S->beta;
    const int warp = (blockIdx.x * BS + threadIdx.x) >> 5, nwarps = gridDim.x * (BS / 32);
    const float loc = bspmv_slices_dir<U, TC>(nbr, nslice, soff, swid, scol, sv, z, odd ? pb : pa, beta, odd ? pa : pb,
                                              q, warp, nwarps);
    const double bsum = block_sum_f(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bsum;
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

// The folded product for few slices: one CTA per slice, its eight warps take
// the slots in turn (at most four each for 27 blocks a row, all their loads
// in flight at once), and the warps' partial rows are added in warp order
// through shared memory.  A warp per slice leaves most SMs idle below a few
// hundred slices and walks its slots one batch after the other.  Bound by
// latency: at 9,261 nodes the iteration took 30.1 us with a warp per slice,
// 25.8 us with this product (22.5 us since the update kernel waits less).
template <typename TC>
__global__ void __launch_bounds__(BS) k_bspmv_dir_split(int nbr, int nslice, const int* __restrict__ soff,
                                                        const int* __restrict__ swid, const TC* __restrict__ scol,
                                                        const float* __restrict__ sv, const float* __restrict__ z,
                                                        float* pa, float* pb, float* __restrict__ q, CGScal* S,
                                                        double* part) {
    if (S->done) return;
    constexpr int U = 4, NWP = BS / 32;
    __shared__ double sh[32];
    __shared__ float acc[NWP][3][32];
    const bool odd = S->iters & 1;
    const float beta = (float)S->beta;
    const float* __restrict__ pold = odd ? pb : pa;
    float* __restrict__ pnew = odd ? pa : pb;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float loc = 0.f;
    for (int s = blockIdx.x; s < nslice; s += gridDim.x) {
        const int i = s * 32 + lane;
        const int o = soff[s], wid = swid[s];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        for (int k = w; k < wid; k += U * NWP) {
            int j[U];
            float v[U][9];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int kk = k + u * NWP;
                if (kk < wid) {
                    j[u] = __ldg(scol + o + kk * 32 + lane) + (sizeof(TC) == 2 ? i : 0);
                    const float* vp = sv + (size_t)((o >> 5) + kk) * 288 + lane;
#pragma unroll
                    for (int e = 0; e < 9; ++e) v[u][e] = __ldg(vp + 32 * e);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (k + u * NWP < wid) {
                    const size_t b = 3 * (size_t)j[u];
                    const float x0 = fmaf(beta, __ldg(pold + b), __ldg(z + b));
                    const float x1 = fmaf(beta, __ldg(pold + b + 1), __ldg(z + b + 1));
                    const float x2 = fmaf(beta, __ldg(pold + b + 2), __ldg(z + b + 2));
                    a0 += v[u][0] * x0 + v[u][1] * x1 + v[u][2] * x2;
                    a1 += v[u][3] * x0 + v[u][4] * x1 + v[u][5] * x2;
                    a2 += v[u][6] * x0 + v[u][7] * x1 + v[u][8] * x2;
                }
            }
        }
        acc[w][0][lane] = a0; acc[w][1][lane] = a1; acc[w][2][lane] = a2;
        __syncthreads();
        if (w < 3 && i < nbr) {  // warp c: component c of the slice's rows
            float t = 0.f;
#pragma unroll
            for (int k = 0; k < NWP; ++k) t += acc[k][w][lane];
            const size_t b = 3 * (size_t)i + w;
            const float p = fmaf(beta, __ldg(pold + b), __ldg(z + b));
            pnew[b] = p;
            q[b] = t;
            loc += p * t;
        }
        __syncthreads();
    }
    const double bsum = block_sum_f(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bsum;
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

// q = A p on the block-row CSR copy: LPB lanes per block row
template <int LPB>
__global__ void __launch_bounds__(BS, 8) k_brow_spmv(int nbr, const int* __restrict__ bptr, const int* __restrict__ bcol,
                                                     const float* __restrict__ bv, int nblk, const float* __restrict__ p,
                                                     float* __restrict__ q, CGScal* S, double* part) {
    if (S->done) return;
    __shared__ double sh[32];
    const int lane = threadIdx.x % LPB;
    const int grp = (blockIdx.x * BS + threadIdx.x) / LPB, ngrp = gridDim.x * BS / LPB;
    const int wgrp = grp - grp % (32 / LPB);  // warp-uniform loop (full-mask shuffles below)
    float loc = 0.f;
    for (int base = wgrp; base < nbr; base += ngrp) {
        const int i = base + (grp - wgrp);
        const bool act = i < nbr;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        const int lo = act ? bptr[i] : 0, hi = act ? bptr[i + 1] : 0;
        for (int k = lo + lane; k < hi; k += LPB) {
            const int j = __ldg(bcol + k);
            const float x0 = __ldg(p + 3 * j), x1 = __ldg(p + 3 * j + 1), x2 = __ldg(p + 3 * j + 2);
            a0 += __ldg(bv + k) * x0 + __ldg(bv + (size_t)nblk + k) * x1 + __ldg(bv + 2 * (size_t)nblk + k) * x2;
            a1 += __ldg(bv + 3 * (size_t)nblk + k) * x0 + __ldg(bv + 4 * (size_t)nblk + k) * x1 + __ldg(bv + 5 * (size_t)nblk + k) * x2;
            a2 += __ldg(bv + 6 * (size_t)nblk + k) * x0 + __ldg(bv + 7 * (size_t)nblk + k) * x1 + __ldg(bv + 8 * (size_t)nblk + k) * x2;
        }
#pragma unroll
        for (int o = LPB / 2; o > 0; o >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o, LPB);
            a1 += __shfl_xor_sync(0xffffffffu, a1, o, LPB);
            a2 += __shfl_xor_sync(0xffffffffu, a2, o, LPB);
        }
        if (act && lane == 0) {
            q[3 * i] = a0; q[3 * i + 1] = a1; q[3 * i + 2] = a2;
            loc += p[3 * i] * a0 + p[3 * i + 1] * a1 + p[3 * i + 2] * a2;
        }
    }
    const double bsum = block_sum_f(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bsum;
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

__device__ inline void bj_apply(const float* __restrict__ binv, int nbr, int i, const float r[3], float z[3]) {
    (void)nbr;
#pragma unroll
    for (int a = 0; a < 3; ++a)
        z[a] = binv[(size_t)i * 9 + a * 3] * r[0] + binv[(size_t)i * 9 + a * 3 + 1] * r[1] + binv[(size_t)i * 9 + a * 3 + 2] * r[2];
}

// Block-Jacobi vector kernels, one thread per DOF: a block of 192 threads
// covers 64 whole nodes, so the three residual components of a node are
// exchanged through shared memory and every global access is coalesced.
constexpr int NBS = 192;

// one thread per node: the node's three residual entries, search direction,
// A p and its inverse diagonal block are all loaded at once (no shared-memory
// exchange, no barrier in the data path).  Two blocks per SM stride over the
// nodes: fewer blocks shorten the reduction tail (partials + last-block
// ticket), which dominates a kernel that streams ~30 MB
constexpr int NODE_BS = 256;
static unsigned node_grid(const isl_ctx* c, long long nbr) {
    return (unsigned)std::max<long long>(1, std::min<long long>((nbr + NODE_BS - 1) / NODE_BS, 2LL * c->sm_count));
}
// FZ: the direction update is folded into the SpMV (k_bspmv_dir): p is the
// buffer that product wrote (p2 on even iteration counts, p on odd ones), and
// z = B^-1 r is stored for the next product
template <bool FZ>
__global__ void __launch_bounds__(NODE_BS) k_cg_update_b3n(int nbr, float* __restrict__ x, float* __restrict__ r,
                                                           const float* __restrict__ p1, const float* __restrict__ p2,
                                                           const float* __restrict__ q, const float* __restrict__ binv,
                                                           float* __restrict__ zout, CGScal* S, double* part,
                                                           int max_iter) {
    if (S->done) return;
    __shared__ double sh[32];
    const float* __restrict__ p = (FZ && !(S->iters & 1)) ? p2 : p1;
    const float alpha = (float)S->alpha;
    float rr = 0.f, rz = 0.f;
    for (int i = blockIdx.x * NODE_BS + threadIdx.x; i < nbr; i += gridDim.x * NODE_BS) {
        const size_t d = 3 * (size_t)i;
        float b[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) b[k] = ld(binv + 9 * (size_t)i + k);
        float rv[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            x[d + a] += alpha * ld(p + d + a);
            rv[a] = r[d + a] - alpha * ld(q + d + a);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            r[d + a] = rv[a];
            const float z = b[3 * a] * rv[0] + b[3 * a + 1] * rv[1] + b[3 * a + 2] * rv[2];
            if (FZ) zout[d + a] = z;
            rr += rv[a] * rv[a];
            rz += rv[a] * z;
        }
    }
    // r.r and r.z: block and grid sums in double-float, as in k_bspmv_dir
    df b1, b2;
    block_sum_df2(rr, rz, reinterpret_cast<float*>(sh), b1, b2);
    if (threadIdx.x == 0) reinterpret_cast<float4*>(part)[blockIdx.x] = make_float4(b1.hi, b1.lo, b2.hi, b2.lo);
    if (!last_block(&S->ticket2)) return;
    double trr, trz;
    reduce_parts2_df_blk<NODE_BS>(reinterpret_cast<const float4*>(part), gridDim.x, sh, trr, trz);
    if (threadIdx.x == 0) {
        S->rr = trr;
        S->iters += 1;
        S->absOld = S->absNew;
        S->beta = trz / S->absNew;
        S->absNew = trz;
        if (!(trr == trr) || !(trz == trz)) { S->bad = 1; S->done = 1; }
        else if (trr < S->threshold) S->done = 1;
        else if (trr < S->rrtrig) S->done = 3;
        else if (S->iters >= max_iter) S->done = 2;
        S->ticket2 = 0;
    }
}

// The same update with the node records staged through shared memory: a
// block takes tiles of UT nodes, reads the tile's 3 UT entries of x, r, p, q
// and its 9 UT inverse-block entries with consecutive threads on consecutive
// words (every warp load is 128 contiguous bytes, against 384 B and 1,152 B
// spans of the node-per-thread loads), updates one node per thread from
// shared memory (strides 3 and 9 words: no bank conflicts), and writes x, r
// and z back the same coalesced way.  Per-node arithmetic is that of
// k_cg_update_b3n.
constexpr int UT = 256;
template <bool FZ>
__global__ void __launch_bounds__(UT) k_cg_update_b3t(int nbr, float* __restrict__ x, float* __restrict__ r,
                                                      const float* __restrict__ p1, const float* __restrict__ p2,
                                                      const float* __restrict__ q, const float* __restrict__ binv,
                                                      float* __restrict__ zout, CGScal* S, double* part, int max_iter) {
    if (S->done) return;
    __shared__ float sx[3 * UT], sr[3 * UT], sp[3 * UT], sq[3 * UT], sb[9 * UT];
    __shared__ double sh[32];
    const float* __restrict__ p = (FZ && !(S->iters & 1)) ? p2 : p1;
    const float alpha = (float)S->alpha;
    float rr = 0.f, rz = 0.f;
    const int ntile = (nbr + UT - 1) / UT;
    for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
        const int nn = min(UT, nbr - t * UT);
        const size_t d0 = (size_t)3 * UT * t, b0 = (size_t)9 * UT * t;
        for (int k = threadIdx.x; k < 3 * nn; k += UT) {
            sx[k] = x[d0 + k];
            sr[k] = r[d0 + k];
            sp[k] = __ldg(p + d0 + k);
            sq[k] = __ldg(q + d0 + k);
        }
        for (int k = threadIdx.x; k < 9 * nn; k += UT) sb[k] = __ldg(binv + b0 + k);
        __syncthreads();
        if (threadIdx.x < nn) {
            const int i = threadIdx.x;
            float rv[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                sx[3 * i + a] += alpha * sp[3 * i + a];
                rv[a] = sr[3 * i + a] - alpha * sq[3 * i + a];
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                sr[3 * i + a] = rv[a];
                const float z = sb[9 * i + 3 * a] * rv[0] + sb[9 * i + 3 * a + 1] * rv[1] + sb[9 * i + 3 * a + 2] * rv[2];
                if (FZ) sp[3 * i + a] = z;  // the node's own p entry is consumed: the slot carries z out
                rr += rv[a] * rv[a];
                rz += rv[a] * z;
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < 3 * nn; k += UT) {
            x[d0 + k] = sx[k];
            r[d0 + k] = sr[k];
            if (FZ) zout[d0 + k] = sp[k];
        }
        __syncthreads();
    }
    const double b1 = block_sum_f(rr, sh);
    const double b2 = block_sum_f(rz, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = b1; part[2 * blockIdx.x + 1] = b2; }
    if (!last_block(&S->ticket2)) return;
    double trr, trz;
    reduce_parts2_blk<UT>(part, gridDim.x, sh, trr, trz);
    if (threadIdx.x == 0) {
        S->rr = trr;
        S->iters += 1;
        S->absOld = S->absNew;
        S->beta = trz / S->absNew;
        S->absNew = trz;
        if (!(trr == trr) || !(trz == trz)) { S->bad = 1; S->done = 1; }
        else if (trr < S->threshold) S->done = 1;
        else if (trr < S->rrtrig) S->done = 3;
        else if (S->iters >= max_iter) S->done = 2;
        S->ticket2 = 0;
    }
}

__global__ void __launch_bounds__(NBS) k_cg_dir_b3(int nbr, const float* __restrict__ r, const float* __restrict__ binv,
                                                   float* __restrict__ p, const CGScal* S) {
    if (S->done) return;
    __shared__ float sr[NBS];
    const float beta = (float)S->beta;
    const int n = 3 * nbr;
    for (int base = blockIdx.x * NBS; base < n; base += gridDim.x * NBS) {
        const int d = base + threadIdx.x;
        sr[threadIdx.x] = (d < n) ? r[d] : 0.f;
        __syncthreads();
        if (d < n) {
            const int a = threadIdx.x % 3, n0 = threadIdx.x - a, node = d / 3;
            const float* B = binv + (size_t)node * 9 + a * 3;
            p[d] = B[0] * sr[n0] + B[1] * sr[n0 + 1] + B[2] * sr[n0 + 2] + beta * p[d];
        }
        __syncthreads();
    }
}

// x = 0, r = b, p = 0, absNew = r.B^{-1}r; with restart != 0 only r = r64 and
// beta = (r.z)_new / (r.z)_previous (reliable update)
// Persistent mixed block CG: the iterations (direction, SpMV, update) of
// one chunk run inside a single cooperative launch, with a grid barrier after
// each phase.  Every block sums the partials of all blocks itself, in a fixed
// order, so all blocks hold the same alpha, beta and decisions without a
// ticket; the arithmetic per element is that of k_cg_dir_b3, k_bspmv_batch
// and k_cg_update_b3n.  Vectors written inside the kernel are read with
// ordinary loads, never the non-coherent path.  Block 0 leaves the scalar record as k_cg_update_b3n does (done 1:
// converged, 2: iteration limit, 3: reliable update due, 0: chunk used up).
constexpr int PERSIST_U = 8;
constexpr int PERSIST_CHUNK = 1024;
// below this many nodes the separate kernels are launch-bound and the
// persistent kernel is the faster path; above it the graph path is
constexpr int PERSIST_MAX_NBR = 32768;
__global__ void __launch_bounds__(BS, 2) k_cg_persist_b3(int nbr, int nslice, const int* __restrict__ soff,
                                                         const int* __restrict__ swid, const int* __restrict__ scol,
                                                         const float* __restrict__ sv, const float* __restrict__ binv,
                                                         float* x, float* r, float* p, float* q, CGScal* S, double* part,
                                                         unsigned* bar, int max_iter, int chunk) {
    __shared__ double sh[32];
    __shared__ double bc[2];
    if (S->done) return;
    const int G = gridDim.x;
    double rz = S->absNew, beta = S->beta, rz_old = S->absOld, rr = S->rr;
    int iters = S->iters;
    const double thr = S->threshold, trig = S->rrtrig;
    const int tid = blockIdx.x * BS + threadIdx.x, nthr = G * BS;
    double* ppq = part;      // [G]: p.q per block
    double* prz = part + G;  // [2G]: r.r, r.z per block
    int done = 0, bad = 0;
    for (int step = 0; step < chunk && !done; ++step) {
        // p = B^-1 r + beta p
        const float fb = (float)beta;
        for (int i = tid; i < nbr; i += nthr) {
            const float r0 = r[3 * i], r1 = r[3 * i + 1], r2 = r[3 * i + 2];
            const float* B = binv + 9 * (size_t)i;
#pragma unroll
            for (int a = 0; a < 3; ++a)
                p[3 * i + a] = __ldg(B + 3 * a) * r0 + __ldg(B + 3 * a + 1) * r1 + __ldg(B + 3 * a + 2) * r2 +
                               fb * p[3 * i + a];
        }
        if (!grid_sync(bar, &S->fault)) return;
        // q = A p, p.q
        const float loc = bspmv_slices<PERSIST_U, true>(nbr, nslice, soff, swid, scol, sv, p, q, tid >> 5, nthr >> 5);
        const double bsum = block_sum_f(loc, sh);
        if (threadIdx.x == 0) ppq[blockIdx.x] = bsum;
        if (!grid_sync(bar, &S->fault)) return;
        const double pap = reduce_parts(ppq, G, 1, 0, sh);
        if (threadIdx.x == 0) bc[0] = pap;
        __syncthreads();
        const float alpha = (float)block_div(rz, bc[0]);
        // x += alpha p, r -= alpha q; r.r and r.z with z = B^-1 r
        float frr = 0.f, frz = 0.f;
        for (int i = tid; i < nbr; i += nthr) {
            const float* B = binv + 9 * (size_t)i;
            float b9[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) b9[k] = __ldg(B + k);
            float rv[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int d = 3 * i + a;
                x[d] += alpha * p[d];
                rv[a] = r[d] - alpha * q[d];
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                r[3 * i + a] = rv[a];
                const float z = b9[3 * a] * rv[0] + b9[3 * a + 1] * rv[1] + b9[3 * a + 2] * rv[2];
                frr += rv[a] * rv[a];
                frz += rv[a] * z;
            }
        }
        const double b1 = block_sum_f(frr, sh);
        const double b2 = block_sum_f(frz, sh);
        if (threadIdx.x == 0) { prz[2 * blockIdx.x] = b1; prz[2 * blockIdx.x + 1] = b2; }
        if (!grid_sync(bar, &S->fault)) return;
        double trr, trz;
        reduce_parts2(prz, G, sh, trr, trz);
        if (threadIdx.x == 0) { bc[0] = trr; bc[1] = trz; }
        __syncthreads();
        trr = bc[0];
        trz = bc[1];
        __syncthreads();
        iters += 1;
        rr = trr;
        rz_old = rz;
        beta = block_div(trz, rz);
        rz = trz;
        if (!(trr == trr) || !(trz == trz)) { bad = 1; done = 1; }
        else if (trr < thr) done = 1;
        else if (trr < trig) done = 3;
        else if (iters >= max_iter) done = 2;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S->rr = rr;
        S->iters = iters;
        S->absOld = rz_old;
        S->beta = beta;
        S->absNew = rz;
        if (bad) S->bad = 1;
        S->done = done;
    }
}

// blocks of the persistent kernel: as many as can be resident (at most two
// per SM), 0 where cooperative launches are unavailable
static int persist_grid(isl_ctx* c) {
    if (c->persist_grid >= 0) return c->persist_grid;
    int coop = 0, nb = 0;
    c->persist_grid = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) == cudaSuccess && coop &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_cg_persist_b3, BS, 0) == cudaSuccess && nb > 0)
        c->persist_grid = std::min(nb, 2) * c->sm_count;
    cudaGetLastError();
    return c->persist_grid;
}

// zout (may be null): z = B^-1 r is stored for a folded direction update;
// aeq (may be null): padded blocks, b is indexed by equation through aeq
// (zero at constrained components)
// restart == 2: a reliable update after which the FP32 directions restart
// (beta = 0): the true residual has not dropped since the previous update
__global__ void __launch_bounds__(BS) k_cg_init_b3(int nbr, const double* __restrict__ b, const int* __restrict__ aeq,
                                                   float* __restrict__ x, float* __restrict__ r,
                                                   float* __restrict__ p, const float* __restrict__ binv, float* __restrict__ zout,
                                                   CGScal* S, double* part, double tol, int restart, double trig) {
    __shared__ double sh[32];
    double bb = 0.0, bz = 0.0;
    for (int i = blockIdx.x * BS + threadIdx.x; i < nbr; i += gridDim.x * BS) {
        float ri[3], zi[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int e = aeq ? aeq[3 * i + a] : 3 * i + a;
            const double bi = e >= 0 ? b[e] : 0.0;
            ri[a] = (float)bi;
            r[3 * i + a] = ri[a];
            if (!restart) { x[3 * i + a] = 0.f; p[3 * i + a] = 0.f; bb += bi * bi; }
            else bb += (double)ri[a] * (double)ri[a];
        }
        bj_apply(binv, nbr, i, ri, zi);
        if (zout) { zout[3 * i] = zi[0]; zout[3 * i + 1] = zi[1]; zout[3 * i + 2] = zi[2]; }
        bz += (double)ri[0] * zi[0] + (double)ri[1] * zi[1] + (double)ri[2] * zi[2];
    }
    const double b1 = block_sum(bb, sh);
    const double b2 = block_sum(bz, sh);
    if (threadIdx.x == 0) { part[2 * blockIdx.x] = b1; part[2 * blockIdx.x + 1] = b2; }
    if (last_block(&S->ticket2)) {
        double tbb, tbz;
        reduce_parts2(part, gridDim.x, sh, tbb, tbz);
        if (threadIdx.x == 0) {
            if (!restart) {
                S->rhsNorm2 = tbb;
                S->threshold = tol * tol * tbb;
                S->rrtrig = trig * tbb;
                S->absNew = tbz;
                S->absOld = tbz;
                S->beta = 0.0;
                S->rr = tbb;
                S->iters = 0;
                S->bad = !(tbb == tbb);
                S->done = (tbb == 0.0 || tbb < S->threshold || S->bad) ? 1 : 0;
                S->ticket1 = 0;
            } else {
                S->rr = tbb;
                S->beta = restart == 2 ? 0.0 : tbz / S->absOld;
                S->absNew = tbz;
                S->rrtrig = trig;
                S->done = 0;
            }
            S->ticket2 = 0;
        }
    }
}

static unsigned sell_grid(isl_ctx* c) {
    const long long need = (c->nslice + (BS / 32) - 1) / (BS / 32);
    return (unsigned)std::max<long long>(1, std::min<long long>(need, (long long)c->sm_count * (2048 / BS)));
}

// kind 1..3: sliced-ELL with slice-loop unroll 1, 2, 4; kind 5..7: sliced-ELL
// with the loads of 2, 4, 8 slots batched; kind 4, 8, 16: block-row CSR with
// that many lanes per block row
static void launch_bspmv(int kind, unsigned grid, cudaStream_t st, isl_ctx* c, const float* p, float* q, CGScal* S, double* part) {
    (void)grid;
    const int nbr = (int)c->nbr, ns = (int)c->nslice, nb = (int)c->nblk;
    const unsigned g = sell_grid(c), gv = vec_grid(c);
    switch (kind) {
        case 1: k_bspmv_pap<1><<<g, BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, c->nslot, p, q, S, part); break;
        case 3: k_bspmv_pap<4><<<g, BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, c->nslot, p, q, S, part); break;
        case 5: k_bspmv_batch<2, 4><<<std::min(g, 4u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, p, q, S, part); break;
        case 6: k_bspmv_batch<4, 3><<<std::min(g, 3u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, p, q, S, part); break;
        case 7: k_bspmv_batch<8, 2><<<std::min(g, 2u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, p, q, S, part); break;
        case 4: k_brow_spmv<4><<<gv, BS, 0, st>>>(nbr, c->dbptr.p, c->dbcol.p, c->dbval.p, nb, p, q, S, part); break;
        case 8: k_brow_spmv<8><<<gv, BS, 0, st>>>(nbr, c->dbptr.p, c->dbcol.p, c->dbval.p, nb, p, q, S, part); break;
        case 16: k_brow_spmv<16><<<gv, BS, 0, st>>>(nbr, c->dbptr.p, c->dbcol.p, c->dbval.p, nb, p, q, S, part); break;
        default: k_bspmv_pap<2><<<g, BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, c->dscol.p, c->dsval.p, c->nslot, p, q, S, part); break;
    }
}

// the batched-load kinds 5..7 also exist with the direction update folded in
static bool bspmv_dir_kind(int kind) { return kind >= 5 && kind <= 7; }
template <typename TC>
static void launch_bspmv_dir_t(int kind, cudaStream_t st, isl_ctx* c, const TC* scol, const float* z, float* pa,
                               float* pb, float* q, CGScal* S, double* part) {
    const int nbr = (int)c->nbr, ns = (int)c->nslice;
    const unsigned g = sell_grid(c);
    if (kind == 9) {
        k_bspmv_dir_split<TC><<<(unsigned)std::min<long long>(c->nslice, 4LL * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, scol, c->dsval.p, z, pa, pb, q, S, part);
        return;
    }
    switch (kind) {
        case 5: k_bspmv_dir<2, 4, TC><<<std::min(g, 4u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, scol, c->dsval.p, z, pa, pb, q, S, part); break;
        case 6: k_bspmv_dir<4, 3, TC><<<std::min(g, 3u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, scol, c->dsval.p, z, pa, pb, q, S, part); break;
        default: k_bspmv_dir<8, 2, TC><<<std::min(g, 2u * c->sm_count), BS, 0, st>>>(nbr, ns, c->dsoff.p, c->dswid.p, scol, c->dsval.p, z, pa, pb, q, S, part); break;
    }
}
// the 16-bit column offsets where the matrix has them (and ISL_OPT_SHORT_COLUMNS allows)
static void launch_bspmv_dir(int kind, cudaStream_t st, isl_ctx* c, const float* z, float* pa, float* pb, float* q,
                             CGScal* S, double* part) {
    if (c->scol16 && c->use_scol16) launch_bspmv_dir_t<short>(kind, st, c, c->dscol16.p, z, pa, pb, q, S, part);
    else launch_bspmv_dir_t<int>(kind, st, c, c->dscol.p, z, pa, pb, q, S, part);
}

// autotune of the block SpMV (format and row mapping) on the current matrix
// The variants launch different grids, so the p.q partial sums, and with them
// the rounding of alpha, follow the choice: a different variant moves the CG
// iteration count by a few percent.  To keep the choice, and the iteration
// count, the same from run to run despite timing noise, the candidates are
// ranked in a fixed preference order and the first within 2 % of the fastest
// is taken.
static int autotune_lpb(isl_ctx* c, const float* p, float* q, CGScal* S, double* part) {
    const int cand[9] = {7, 6, 5, 1, 2, 3, 4, 8, 16};  // preference order
    if (c->nbr < 8000) return 2;
    int cached = 0;
    if (tune_lookup(c, "bspmv", &cached) && std::find(cand, cand + 9, cached) != cand + 9) return cached;
    float ms_of[9];
    float bestms = 1e30f;
    cudaMemsetAsync(S, 0, sizeof(CGScal), c->stream);
    c->launches += 9 * 21;
    for (int k = 0; k < 9; ++k) {
        launch_bspmv(cand[k], 0, c->stream, c, p, q, S, part);
        cudaEventRecord(c->ev[2], c->stream);
        for (int r = 0; r < 20; ++r) launch_bspmv(cand[k], 0, c->stream, c, p, q, S, part);
        cudaEventRecord(c->ev[3], c->stream);
        cudaEventSynchronize(c->ev[3]);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev[2], c->ev[3]);
        ms_of[k] = ms;
        bestms = std::min(bestms, ms);
    }
    int best = cand[0];
    for (int k = 0; k < 9; ++k)
        if (ms_of[k] <= 1.02f * bestms) { best = cand[k]; break; }
    tune_store(c, "bspmv", best);
    return best;
}

bool update_kind_valid(int k) { return k == 1 || k == 2 || k == 4 || k == 8; }

// constant fill (timing inputs)
__global__ void k_fill(int64_t n, float* __restrict__ a, float v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) a[i] = v;
}
__global__ void k_fill64(int64_t n, double* __restrict__ a, double v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) a[i] = v;
}

// update kernel of the block CG: 1 one thread per node (k_cg_update_b3n, two
// blocks per SM); 2, 4, 8: tiles of UT nodes staged through shared memory
// (k_cg_update_b3t) with that many blocks per SM
static void launch_update(isl_ctx* c, int kind, bool fz, cudaStream_t st, float* x, float* r, const float* p1,
                          const float* p2, const float* q, float* z, CGScal* S, int mi) {
    const int nbr = (int)c->nbr;
    if (kind <= 1) {
        const unsigned g = node_grid(c, nbr);
        if (fz) k_cg_update_b3n<true><<<g, NODE_BS, 0, st>>>(nbr, x, r, p1, p2, q, c->dbinv.p, z, S, c->dpart.p, mi);
        else k_cg_update_b3n<false><<<g, NODE_BS, 0, st>>>(nbr, x, r, p1, p2, q, c->dbinv.p, z, S, c->dpart.p, mi);
        return;
    }
    const long long ntile = (nbr + UT - 1) / UT;
    const unsigned g = (unsigned)std::max<long long>(1, std::min<long long>(ntile, (long long)kind * c->sm_count));
    if (fz) k_cg_update_b3t<true><<<g, UT, 0, st>>>(nbr, x, r, p1, p2, q, c->dbinv.p, z, S, c->dpart.p, mi);
    else k_cg_update_b3t<false><<<g, UT, 0, st>>>(nbr, x, r, p1, p2, q, c->dbinv.p, z, S, c->dpart.p, mi);
}

// detect the node-blocked structure and build the block pattern (setup)
// padded node blocks (some DOF objects partly constrained): the equation map
// of the block rows from the host numbering, then the block pattern on the
// device (k_bsr_pattern_pad); false when the pattern is not of that form
static int block_pattern_pad(isl_ctx* c, bool* ok) {
    *ok = false;
    const int64_t ndo = c->ndofobj, n = c->neq;
    std::vector<int32_t> aeq, eqblk((size_t)n, -1);
    aeq.reserve((size_t)3 * ndo);
    int64_t nbr = 0, next = 0;
    for (int64_t o = 0; o < ndo; ++o) {
        const int32_t* q = &c->heq[(size_t)o * 3];
        if (q[0] < 0 && q[1] < 0 && q[2] < 0) continue;
        for (int a = 0; a < 3; ++a) {
            if (q[a] < 0) continue;
            if (q[a] != next) return ISL_OK;  // equations not consecutive per object
            eqblk[(size_t)q[a]] = (int32_t)nbr;
            ++next;
        }
        aeq.insert(aeq.end(), q, q + 3);
        ++nbr;
    }
    if (next != n || nbr == 0) return ISL_OK;
    cudaStream_t st = c->stream;
    DBuf<int32_t> deqblk, cnt;
    ISL_CHECK_CUDA(c, c->dbaeq.alloc((size_t)3 * nbr));
    ISL_CHECK_CUDA(c, deqblk.alloc((size_t)n));
    ISL_CHECK_CUDA(c, cnt.alloc((size_t)nbr));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dbaeq.p, aeq.data(), aeq.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(deqblk.p, eqblk.data(), eqblk.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dflags.p + 1, 0, sizeof(int), st));
    k_bsr_pattern_pad<<<vec_grid(c), BS, 0, st>>>((int)nbr, 0, c->dbaeq.p, deqblk.p, c->drowptr.p, c->dcolind.p, cnt.p,
                                                  nullptr, nullptr, nullptr, nullptr, c->dflags.p + 1);
    int bad = 0;
    std::vector<int32_t> hc((size_t)nbr), bp((size_t)nbr + 1, 0);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(&bad, c->dflags.p + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hc.data(), cnt.p, hc.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    c->launches += 1;
    if (bad) return ISL_OK;
    int64_t tot = 0;
    for (int64_t i = 0; i < nbr; ++i) { bp[(size_t)i] = (int32_t)tot; tot += hc[(size_t)i]; }
    if (tot >= INT32_MAX / 9) return ISL_OK;
    bp[(size_t)nbr] = (int32_t)tot;
    c->nbr = nbr;
    c->nblk = tot;
    ISL_CHECK_CUDA(c, c->dbptr.alloc(nbr + 1));
    ISL_CHECK_CUDA(c, c->dbcol.alloc(c->nblk));
    ISL_CHECK_CUDA(c, c->dbrow.alloc(c->nblk));
    ISL_CHECK_CUDA(c, c->dbcb.alloc(c->nblk));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dbptr.p, bp.data(), bp.size() * 4, cudaMemcpyHostToDevice, st));
    k_bsr_pattern_pad<<<vec_grid(c), BS, 0, st>>>((int)nbr, 1, c->dbaeq.p, deqblk.p, c->drowptr.p, c->dcolind.p, cnt.p,
                                                  c->dbptr.p, c->dbcol.p, c->dbrow.p, c->dbcb.p, c->dflags.p + 1);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    c->launches += 1;
    *ok = true;
    return ISL_OK;
}

int block_pattern(isl_ctx* c, const std::vector<int32_t>& rp) {
    c->blocked = false;
    c->bpad = false;
    c->dbaeq.release();
    c->dbcb.release();
    if (c->ncomp != 3 || c->ninst > 1) return ISL_OK;
    bool uniform = c->neq % 3 == 0;
    for (int64_t o = 0; uniform && o < c->ndofobj; ++o) {
        const uint8_t s0 = c->status[(size_t)o * 3];
        if (c->status[(size_t)o * 3 + 1] != s0 || c->status[(size_t)o * 3 + 2] != s0) uniform = false;
    }
    if (uniform) {
        const int64_t nbr = c->neq / 3;
        for (int64_t i = 0; i < nbr; ++i) {
            const int32_t len = rp[3 * i + 1] - rp[3 * i];
            if (rp[3 * i] % 9 || len % 3 || rp[3 * i + 2] - rp[3 * i + 1] != len || rp[3 * i + 3] - rp[3 * i + 2] != len) return ISL_OK;
        }
        c->nbr = nbr;
        c->nblk = c->nnz / 9;
        ISL_CHECK_CUDA(c, c->dbptr.alloc(nbr + 1));
        ISL_CHECK_CUDA(c, c->dbcol.alloc(c->nblk));
        ISL_CHECK_CUDA(c, c->dbrow.alloc(c->nblk));
        ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dflags.p + 1, 0, sizeof(int), c->stream));
        k_bsr_pattern<<<vec_grid(c), BS, 0, c->stream>>>((int)nbr, c->drowptr.p, c->dcolind.p, c->dbptr.p, c->dbcol.p, c->dbrow.p,
                                                         c->dflags.p + 1);
        int bad = 0;
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(&bad, c->dflags.p + 1, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
        c->launches += 1;
        c->blocked = (bad == 0);
    } else {
        bool ok = false;
        const int rc = block_pattern_pad(c, &ok);
        if (rc != ISL_OK) return rc;
        c->blocked = c->bpad = ok;
        if (!ok) { c->dbaeq.release(); c->dbcb.release(); }
    }
    c->bsr_serial = -1;
    c->bspmv_lpb = 0;
    c->bupd_kind[0] = c->bupd_kind[1] = 0;
    if (!c->blocked) return ISL_OK;
    const int64_t nbr = c->nbr;
    // sliced-ELL layout
    c->nslice = (nbr + 31) / 32;
    ISL_CHECK_CUDA(c, c->dswid.alloc(c->nslice));
    ISL_CHECK_CUDA(c, c->dsoff.alloc(c->nslice + 1));
    k_sell_width<<<vec_grid(c), BS, 0, c->stream>>>((int)nbr, (int)c->nslice, c->dbptr.p, c->dswid.p);
    std::vector<int32_t> wid(c->nslice), off(c->nslice + 1, 0);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(wid.data(), c->dswid.p, wid.size() * 4, cudaMemcpyDeviceToHost, c->stream));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    int64_t tot = 0;
    for (int64_t s2 = 0; s2 < c->nslice; ++s2) { off[s2] = (int32_t)tot; tot += (int64_t)wid[s2] * 32; }
    if (tot >= INT32_MAX) { c->blocked = false; return ISL_OK; }
    off[c->nslice] = (int32_t)tot;
    c->nslot = tot;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dsoff.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, c->stream));
    ISL_CHECK_CUDA(c, c->dscol.alloc(tot));
    ISL_CHECK_CUDA(c, c->dsdst.alloc(c->nblk));
    k_sell_fill<<<vec_grid(c), BS, 0, c->stream>>>((int)nbr, (int)c->nslice, c->dbptr.p, c->dbcol.p, c->dsoff.p, c->dswid.p,
                                                   c->dscol.p, c->dsdst.p);
    {
        // 16-bit column offsets, when every slot's column is within +-32,767
        // block rows of its own (padding rows past nbr point at the last row)
        c->scol16 = false;
        ISL_CHECK_CUDA(c, c->dscol16.alloc(tot));
        ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dflags.p + 1, 0, sizeof(int), c->stream));
        k_sell_col16<<<vec_grid(c), BS, 0, c->stream>>>((int)nbr, (int)c->nslice, c->dsoff.p, c->dswid.p, c->dscol.p,
                                                        c->dscol16.p, c->dflags.p + 1);
        int far = 0;
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(&far, c->dflags.p + 1, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
        c->launches += 1;
        c->scol16 = far == 0;
        if (!c->scol16) c->dscol16.release();
    }
    ISL_CHECK_CUDA(c, c->dsval.alloc((size_t)9 * tot));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dsval.p, 0, (size_t)9 * tot * 4, c->stream));
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    c->launches += 2;
    return ISL_OK;
}

// column ids of the scalar sliced-ELL slots (padding: the row's own column,
// or column 0 in a padding row) and the first slot of every row
__global__ void k_ssell_fill(int nslice, const int* __restrict__ rowptr, const int* __restrict__ colind,
                             const int* __restrict__ soff, const int* __restrict__ swid, const int* __restrict__ srow,
                             int* __restrict__ scol, int* __restrict__ spos) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nslice * 32; i += gridDim.x * blockDim.x) {
        const int s = i / 32, l = i % 32;
        const int row = srow[i];
        const int o = soff[s] + l, w = swid[s];
        const int lo = row >= 0 ? rowptr[row] : 0;
        const int len = row >= 0 ? rowptr[row + 1] - lo : 0;
        if (row >= 0) spos[row] = o;
        for (int k = 0; k < w; ++k) scol[o + k * 32] = k < len ? colind[lo + k] : (row >= 0 ? row : 0);
    }
}

// 16-bit copy of the scalar sliced-ELL columns as offsets from each lane's
// row (row 0 for a padding lane, whose slots hold column 0); any offset
// outside the 16-bit range sets *far
__global__ void k_ssell_col16(int nslice, const int* __restrict__ srow, const int* __restrict__ soff,
                              const int* __restrict__ swid, const int* __restrict__ scol, short* __restrict__ scol16,
                              int* __restrict__ far) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nslice * 32; t += gridDim.x * blockDim.x) {
        const int s = t / 32, l = t % 32;
        const int base = max(srow[t], 0);
        const int o = soff[s] + l, w = swid[s];
        for (int k = 0; k < w; ++k) {
            const int off = scol[o + k * 32] - base;
            if (off < -32767 || off > 32767) { atomicOr(far, 1); scol16[o + k * 32] = 0; }
            else scol16[o + k * 32] = (short)off;
        }
    }
}

// the 16-bit column copy of the scalar sliced-ELL layout, when every offset fits
static int build_ssell16(isl_ctx* c) {
    c->ss16 = false;
    c->dss_col16.release();
    if (c->ss_nslot == 0) return ISL_OK;
    cudaStream_t st = c->stream;
    ISL_CHECK_CUDA(c, c->dss_col16.alloc(c->ss_nslot));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dflags.p + 1, 0, sizeof(int), st));
    k_ssell_col16<<<vec_grid(c), BS, 0, st>>>((int)c->ss_nslice, c->dss_row.p, c->dss_off.p, c->dss_wid.p, c->dss_col.p,
                                              c->dss_col16.p, c->dflags.p + 1);
    int far = 0;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(&far, c->dflags.p + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    c->launches += 1;
    c->ss16 = far == 0;
    if (!c->ss16) c->dss_col16.release();
    return ISL_OK;
}

// Scalar sliced-ELL copy of a system that is not node-blocked (setup).  Rows
// are sorted by length, longest first and stably, within windows of 2048 rows
// (a multiple of 32, so no slice spans two windows); the sort keeps the
// padding near zero while the rows of a slice stay within 2048 of each other,
// so the gathers of p keep their locality.  Batched systems are left out.
int scalar_sell_pattern(isl_ctx* c, const std::vector<int32_t>& rp) {
    c->ss_nslice = c->ss_nslot = 0;
    c->ss_serial = -1;
    c->dss_off.release(); c->dss_wid.release(); c->dss_row.release();
    c->dss_col.release(); c->dss_pos.release(); c->dss_val.release();
    const int64_t n = c->neq;
    if (c->blocked || c->ninst > 1 || n < 20000) return ISL_OK;
    constexpr int64_t WIN = 2048;
    const int64_t nslice = (n + 31) / 32;
    std::vector<int32_t> row((size_t)nslice * 32, -1), wid((size_t)nslice), off((size_t)nslice + 1);
    std::vector<int32_t> idx;
    for (int64_t w0 = 0; w0 < n; w0 += WIN) {
        const int64_t w1 = std::min(n, w0 + WIN);
        idx.resize((size_t)(w1 - w0));
        for (int64_t i = w0; i < w1; ++i) idx[(size_t)(i - w0)] = (int32_t)i;
        std::stable_sort(idx.begin(), idx.end(),
                         [&](int32_t a, int32_t b) { return rp[a + 1] - rp[a] > rp[b + 1] - rp[b]; });
        for (int64_t i = w0; i < w1; ++i) row[(size_t)i] = idx[(size_t)(i - w0)];
    }
    int64_t tot = 0;
    for (int64_t s = 0; s < nslice; ++s) {
        int32_t w = 0;
        for (int l = 0; l < 32; ++l) {
            const int32_t r = row[(size_t)(s * 32 + l)];
            if (r >= 0) w = std::max(w, rp[r + 1] - rp[r]);
        }
        wid[(size_t)s] = w;
        off[(size_t)s] = (int32_t)tot;
        tot += (int64_t)w * 32;
        if (tot >= INT32_MAX) return ISL_OK;  // too large for 32-bit slots: CSR only
    }
    off[(size_t)nslice] = (int32_t)tot;
    cudaStream_t st = c->stream;
    ISL_CHECK_CUDA(c, c->dss_off.alloc(nslice + 1));
    ISL_CHECK_CUDA(c, c->dss_wid.alloc(nslice));
    ISL_CHECK_CUDA(c, c->dss_row.alloc(nslice * 32));
    ISL_CHECK_CUDA(c, c->dss_pos.alloc(n));
    ISL_CHECK_CUDA(c, c->dss_col.alloc(tot));
    ISL_CHECK_CUDA(c, c->dss_val.alloc(tot));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_off.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_wid.p, wid.data(), wid.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_row.p, row.data(), row.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dss_val.p, 0, (size_t)tot * 4, st));
    k_ssell_fill<<<vec_grid(c), BS, 0, st>>>((int)nslice, c->drowptr.p, c->dcolind.p, c->dss_off.p, c->dss_wid.p,
                                             c->dss_row.p, c->dss_col.p, c->dss_pos.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));  // the host vectors above go out of scope
    c->launches += 1;
    c->ss_nslice = nslice;
    c->ss_nslot = tot;
    return build_ssell16(c);
}

// Sliced-ELL copy of a batch of instances (setup): each row block of the
// batched solver (at most 2048 rows of one instance) is a sort window, so its
// slices never mix instances; s0/s1 return the slice range of every block.
// Needs 32-bit slot offsets; otherwise no copy is built (CSR only).
int batch_sell_pattern(isl_ctx* c, const std::vector<int32_t>& b0, const std::vector<int32_t>& b1,
                       std::vector<int32_t>& s0, std::vector<int32_t>& s1) {
    c->ss_nslice = c->ss_nslot = 0;
    c->ss_serial = -1;
    const int64_t n = c->neq;
    std::vector<int32_t> rp((size_t)n + 1);
    cudaStream_t st = c->stream;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(rp.data(), c->drowptr.p, rp.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    const size_t nb = b0.size();
    s0.assign(nb, 0);
    s1.assign(nb, 0);
    std::vector<int32_t> row, wid, off;
    std::vector<int32_t> idx;
    int64_t tot = 0;
    for (size_t b = 0; b < nb; ++b) {
        const int32_t r0 = b0[b], r1 = b1[b];
        s0[b] = (int32_t)wid.size();
        idx.resize((size_t)(r1 - r0));
        for (int32_t i = r0; i < r1; ++i) idx[(size_t)(i - r0)] = i;
        std::stable_sort(idx.begin(), idx.end(), [&](int32_t a, int32_t bb) { return rp[a + 1] - rp[a] > rp[bb + 1] - rp[bb]; });
        for (size_t k = 0; k < idx.size(); k += 32) {
            int32_t w = 0;
            for (size_t l = 0; l < 32; ++l) {
                const int32_t r = k + l < idx.size() ? idx[k + l] : -1;
                row.push_back(r);
                if (r >= 0) w = std::max(w, rp[r + 1] - rp[r]);
            }
            wid.push_back(w);
            off.push_back((int32_t)tot);
            tot += (int64_t)w * 32;
            if (tot >= INT32_MAX) { s0.clear(); s1.clear(); return ISL_OK; }
        }
        s1[b] = (int32_t)wid.size();
    }
    const int64_t nslice = (int64_t)wid.size();
    if (nslice == 0) return ISL_OK;
    off.push_back((int32_t)tot);
    ISL_CHECK_CUDA(c, c->dss_off.alloc(nslice + 1));
    ISL_CHECK_CUDA(c, c->dss_wid.alloc(nslice));
    ISL_CHECK_CUDA(c, c->dss_row.alloc(nslice * 32));
    ISL_CHECK_CUDA(c, c->dss_pos.alloc(n));
    ISL_CHECK_CUDA(c, c->dss_col.alloc(tot));
    ISL_CHECK_CUDA(c, c->dss_val.alloc(tot));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_off.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_wid.p, wid.data(), wid.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->dss_row.p, row.data(), row.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dss_val.p, 0, (size_t)tot * 4, st));
    k_ssell_fill<<<vec_grid(c), BS, 0, st>>>((int)nslice, c->drowptr.p, c->dcolind.p, c->dss_off.p, c->dss_wid.p,
                                             c->dss_row.p, c->dss_col.p, c->dss_pos.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    c->launches += 1;
    c->ss_nslice = nslice;
    c->ss_nslot = tot;
    return build_ssell16(c);
}

// refresh the block values and the block-Jacobi inverses after an assembly
static int ensure_bsr(isl_ctx* c) {
    if (c->bsr_serial == c->asm_serial) return ISL_OK;
    ISL_CHECK_CUDA(c, c->dbinv.alloc((size_t)9 * c->nbr));
    ISL_CHECK_CUDA(c, c->dbval.alloc((size_t)9 * c->nblk));
    const unsigned grid = vec_grid(c);
    if (c->bvals_serial != c->asm_serial) {  // block copies from the FP32 CSR values
        const int rc = ensure_val32(c);
        if (rc != ISL_OK) return rc;
        if (c->bpad)
            k_bsr_values_pad<<<grid, BS, 0, c->stream>>>((int)c->nblk, c->dbrow.p, c->dbcol.p, c->dbcb.p, c->dbaeq.p,
                                                         c->drowptr.p, c->dval32.p, c->dsdst.p, c->dsval.p, c->dbval.p);
        else
            k_bsr_values<<<grid, BS, 0, c->stream>>>((int)c->nblk, c->dbrow.p, c->dbptr.p, c->drowptr.p, c->dval32.p,
                                                     c->dsdst.p, c->dsval.p, c->dbval.p);
        c->launches += 1;
    }
    if (c->bpad) {
        if (c->have64)
            k_block_jacobi_pad<double><<<grid, BS, 0, c->stream>>>((int)c->nbr, c->dbaeq.p, c->ddiag.p, c->dval64.p, c->dbinv.p);
        else
            k_block_jacobi_pad<float><<<grid, BS, 0, c->stream>>>((int)c->nbr, c->dbaeq.p, c->ddiag.p, c->dval32.p, c->dbinv.p);
    } else if (c->have64) {
        k_block_jacobi<double><<<grid, BS, 0, c->stream>>>((int)c->nbr, c->drowptr.p, c->ddiag.p, c->dval64.p, c->dbinv.p);
    } else {
        k_block_jacobi<float><<<grid, BS, 0, c->stream>>>((int)c->nbr, c->drowptr.p, c->ddiag.p, c->dval32.p, c->dbinv.p);
    }
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 1;
    c->bsr_serial = c->asm_serial;
    return ISL_OK;
}

// mixed solve on the block copy: FP32 block-Jacobi CG with FP64 reliable
// updates; without the FP64 matrix, plain FP32 block-Jacobi CG to the
// tolerance on its recursive residual (inexact Newton tangents).  The FP32
// vectors have 3 nbr entries: the equations themselves, or with padded blocks
// the block rows' components (zero where constrained), mapped to equations
// when the right-hand side comes in and the increment goes out.
static int solve_mixed_b3(isl_ctx* c, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* nc) {
    int rc = ensure_bsr(c);
    if (rc != ISL_OK) return rc;
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq;
    const int nbr = (int)c->nbr;
    const size_t na = (size_t)3 * nbr;
    const int* aeq = c->bpad ? c->dbaeq.p : nullptr;
    const bool exact64 = c->have64;
    double* W = c->w64.p;
    double *x64 = W, *r64 = W + n;
    float* V = c->w32.p;
    float *x32 = V, *r32 = V + na, *p32 = V + 2 * na, *q32 = V + 3 * na;
    if (!c->bspmv_lpb) {
        ISL_CHECK_CUDA(c, cudaMemsetAsync(p32, 0, na * 4, st));
        c->bspmv_lpb = autotune_lpb(c, p32, q32, c->dscal.p, c->dpart.p);
    }
    if (exact64 && !c->spmv_lpr64)
        c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, c->drhs.p, W + 3 * n, c->dscal.p, c->dpart.p);
    const int mi = (int)std::min<int64_t>(max_iter, INT32_MAX - 1);
    const unsigned grid = vec_grid(c);
    CGScal* S = c->dscal.p;
    double* dres = (double*)(c->dscal.p + 1);
    unsigned* ticket = &(c->dscal.p + 1)->ticket1;
    const bool want_persist = c->use_persist == 2 || (c->use_persist == 1 && nbr <= PERSIST_MAX_NBR);
    const int pgrid = want_persist ? persist_grid(c) : 0;
    // folded direction update: z = B^-1 r and the second direction buffer
    // take the two spare FP32 vectors of the work area
    const bool fused = pgrid == 0 && c->fuse_dir && bspmv_dir_kind(c->bspmv_lpb);
    float *z32 = fused ? V + 4 * na : nullptr, *p32b = V + 5 * na;
    // update kernel: one thread per node unless ISL_OPT_BLOCK_UPDATE picks a
    // tiled one (timed alone, with its vectors in L2, the tiled kernels can
    // look faster; inside the solve, after the SpMV has streamed the matrix
    // through L2, they are slower at 64^3)
    const int ukind = c->bupd_kind[fused ? 1 : 0] ? c->bupd_kind[fused ? 1 : 0] : 1;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dscal.p, 0, 2 * sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(x64, 0, n * 8, st));
    k_cg_init_b3<<<grid, BS, 0, st>>>(nbr, c->drhs.p, aeq, x32, r32, p32, c->dbinv.p, z32, S, c->dpart.p, tol, 0,
                                      exact64 ? c->ru_drop2 : 0.0);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 1;
    cudaGraph_t graph;
    cudaGraphExec_t exec = nullptr;
    if (pgrid == 0) {
    // DOF-linear vector kernels: one wave of 192-thread blocks
    ISL_CHECK_CUDA(c, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    const unsigned nbd = (unsigned)std::max<long long>(1, (3LL * nbr + NBS - 1) / NBS);  // one pass, no reduction
    for (int k = 0; k < CHUNK; ++k) {
        if (fused) {
            launch_bspmv_dir(c->bspmv_lpb, st, c, z32, p32, p32b, q32, S, c->dpart.p);
            launch_update(c, ukind, true, st, x32, r32, p32, p32b, q32, z32, S, mi);
        } else {
            k_cg_dir_b3<<<nbd, NBS, 0, st>>>(nbr, r32, c->dbinv.p, p32, S);
            launch_bspmv(c->bspmv_lpb, grid, st, c, p32, q32, S, c->dpart.p);
            launch_update(c, ukind, false, st, x32, r32, p32, p32, q32, nullptr, S, mi);
        }
    }
    ISL_CHECK_CUDA(c, cudaStreamEndCapture(st, &graph));
    {
        cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        ISL_CHECK_CUDA(c, e);
    }
    }
    int p_nslice = (int)c->nslice, p_chunk = PERSIST_CHUNK;
    const int* p_soff = c->dsoff.p;
    const int* p_swid = c->dswid.p;
    const int* p_scol = c->dscol.p;
    const float* p_sv = c->dsval.p;
    const float* p_binv = c->dbinv.p;
    double* p_part = c->dpart.p;
    unsigned* p_bar = c->dbar.p;
    int p_nbr = nbr, p_mi = mi;
    void* pargs[] = {&p_nbr, &p_nslice, &p_soff, &p_swid, &p_scol, &p_sv, &p_binv, &x32, &r32, &p32, &q32, &S, &p_part,
                     &p_bar, &p_mi, &p_chunk};
    rc = read_scal(c);
    const double bnorm2 = c->hscal->rhsNorm2;
    double rr_true = bnorm2;
    double rr_last = 0.0;  // true residual of the previous reliable update
    const int64_t max_replays = (int64_t)mi + 64;
    int64_t replays = 0;
    bool converged = (bnorm2 == 0.0);
    while (rc == ISL_OK && !converged) {
        if (++replays > max_replays) { rc = ISL_ERR_TIMEOUT; c->err = "mixed CG made no progress"; break; }
        if (pgrid > 0) {
            // the barrier starts from zero (a barrier that timed out leaves it
            // mid-count); the test hook arms it with an arrival count that the
            // grid never reaches
            const unsigned armed[2] = {0x40000000u, 0u};
            const bool arm = c->barrier_test == 1;
            c->barrier_test = 0;
            if ((arm ? cudaMemcpyAsync(c->dbar.p, armed, sizeof(armed), cudaMemcpyHostToDevice, st)
                     : cudaMemsetAsync(c->dbar.p, 0, 2 * sizeof(unsigned), st)) != cudaSuccess ||
                cudaLaunchCooperativeKernel((const void*)k_cg_persist_b3, dim3(pgrid), dim3(BS), pargs, 0, st) != cudaSuccess) {
                rc = ISL_ERR_CUDA; c->err = "persistent CG launch failed"; break;
            }
            c->launches += 1;
        } else {
            if (cudaGraphLaunch(exec, st) != cudaSuccess) { rc = ISL_ERR_CUDA; c->err = "graph launch failed"; break; }
            c->launches += (fused ? 2 : 3) * CHUNK;
        }
        rc = read_scal(c);
        if (rc != ISL_OK) break;
        const CGScal h = *c->hscal;
        if (h.fault) { rc = ISL_ERR_TIMEOUT; c->err = "persistent CG: a grid barrier timed out"; break; }
        if (h.bad) { rc = ISL_ERR_NAN; c->err = "CG breakdown (non-finite reduction)"; break; }
        const bool at_max = h.iters >= mi;
        if (!(h.done || at_max)) continue;
        if (aeq) k_fold_pad<<<grid, BS, 0, st>>>((int)na, aeq, x32, x64);
        else k_fold<<<grid, BS, 0, st>>>((int)n, x32, x64);
        c->launches += 1;
        if (!exact64) {
            rr_true = h.rr;
            converged = h.done == 1;
            if (!converged) *nc = true;
            break;
        }
        {
            launch_residual(c->spmv_lpr64, grid, st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, x64, c->drhs.p, r64,
                            c->dpart.p, ticket, dres);
            c->launches += 1;
            ISL_CHECK_CUDA(c, cudaMemcpyAsync(&rr_true, dres, 8, cudaMemcpyDeviceToHost, st));
            ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
            if (!(rr_true == rr_true)) { rc = ISL_ERR_NAN; c->err = "refinement residual is not finite"; break; }
            if (rr_true <= tol * tol * bnorm2) { converged = true; break; }
            if (at_max) { *nc = true; break; }
            const int fresh = (rr_last > 0.0 && rr_true >= rr_last) ? 1 : 0;
            rr_last = rr_true;
            k_cg_init_b3<<<grid, BS, 0, st>>>(nbr, r64, aeq, x32, r32, p32, c->dbinv.p, z32, S, c->dpart.p, tol,
                                              fresh ? 2 : 1, c->ru_drop2 * rr_true);
            c->launches += 1;
        }
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (rc != ISL_OK) return rc;
    if (!converged && bnorm2 > 0) *nc = true;
    rc = read_scal(c);
    if (rc != ISL_OK) return rc;
    *iters = c->hscal->iters;
    *rel = bnorm2 > 0 ? std::sqrt(rr_true / bnorm2) : 0.0;
    k_copy64<<<grid, BS, 0, st>>>((int)n, x64, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}

int time_bspmv(isl_ctx* c, int nrep, double* ms) {
    const bool warm = nrep > 0;  // one untimed launch first
    nrep = std::abs(nrep);
    int rc = ensure_work(c);
    if (rc == ISL_OK) rc = ensure_bsr(c);
    if (rc != ISL_OK) return rc;
    const size_t n = (size_t)3 * c->nbr;  // the block space (padded blocks included)
    CGScal* S = c->dscal.p;
    float* V = c->w32.p;
    cudaStream_t st = c->stream;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(S, 0, sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(V + 2 * n, 0, n * 4, st));
    if (!c->bspmv_lpb) c->bspmv_lpb = autotune_lpb(c, V + 2 * n, V + 3 * n, S, c->dpart.p);
    // the product the mixed solve launches: with the direction update folded
    // in where that variant exists (z and the two direction buffers zeroed)
    const bool fused = c->fuse_dir && bspmv_dir_kind(c->bspmv_lpb);
    if (fused) ISL_CHECK_CUDA(c, cudaMemsetAsync(V + 4 * n, 0, 2 * n * 4, st));
    auto one = [&]() {
        if (fused) launch_bspmv_dir(c->bspmv_lpb, st, c, V + 4 * n, V + 2 * n, V + 5 * n, V + 3 * n, S, c->dpart.p);
        else launch_bspmv(c->bspmv_lpb, vec_grid(c), st, c, V + 2 * n, V + 3 * n, S, c->dpart.p);
    };
    if (warm) one();
    cudaEventRecord(c->ev[2], st);
    for (int r = 0; r < nrep; ++r) one();
    cudaEventRecord(c->ev[3], st);
    c->launches += nrep + (warm ? 1 : 0);
    ISL_CHECK_CUDA(c, cudaEventSynchronize(c->ev[3]));
    float t = 0.f;
    cudaEventElapsedTime(&t, c->ev[2], c->ev[3]);
    *ms = t / nrep;
    return ISL_OK;
}

// ===========================================================================
// Two-level solve: the mixed CG with the preconditioner of isl_coarse.cu, for
// node blocks and for scalar systems.  An iteration is the update with the
// local part of the preconditioner, the coarse correction, and the product
// (with the direction update folded in for node blocks, in its own launch
// otherwise).  The reliable updates are decided on the device: every CZ_CHUNK
// iterations the captured graph holds one update's kernels, which return at
// once unless the iteration has stopped for one.  The host only watches for
// the end, one graph launch behind the device.  Eight iterations per update
// slot: a shorter chunk runs the (mostly idle) update kernels more often, a
// longer one idles for longer after a stop.
constexpr int CZ_CHUNK = 8;
// Sizes from which the two-level solve is used: node blocks in one launch, node
// blocks on the graph path (below, the one-level iteration of two launches and
// a few hundred iterations ends as early), equations of scalar systems (below,
// the one-level cluster solve: 7.9 us an iteration).
constexpr int64_t CZ_MIN_NODES_ONE = 64, CZ_MIN_NODES = 1280, CZ_MIN_EQ = 2048;
constexpr int64_t CZ_CLUSTER_ENTRIES = 160000;

__global__ void __launch_bounds__(BS) k_rl_fold(int n, const int* __restrict__ aeq, float* __restrict__ x32,
                                                double* __restrict__ x64, const CGScal* S) {
    if (!S->done || S->fin) return;
    for (int a = blockIdx.x * BS + threadIdx.x; a < n; a += gridDim.x * BS) {
        const int e = aeq ? aeq[a] : a;
        if (e >= 0) x64[e] += (double)x32[a];
        x32[a] = 0.0f;
    }
}

// r64 = b - A64 x64; the last block decides: converged, iteration limit,
// breakdown, or a restart (with new directions when the true residual has not
// dropped since the previous reliable update)
template <int LPR>
__global__ void __launch_bounds__(BS) k_rl_residual(int n, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                                    const double* __restrict__ val, const double* __restrict__ x,
                                                    const double* __restrict__ b, double* __restrict__ r, CGScal* S,
                                                    double* part) {
    if (!S->done || S->fin) return;
    __shared__ double sh[32];
    const int lane = threadIdx.x % LPR;
    const int grp = (blockIdx.x * BS + threadIdx.x) / LPR, ngrp = gridDim.x * BS / LPR;
    const int wgrp = grp - grp % (32 / LPR);
    double loc = 0.0;
    for (int base = wgrp; base < n; base += ngrp) {
        const int row = base + (grp - wgrp);
        const bool act = row < n;
        const double ax = row_dot<double, double, LPR>(row, act, rowptr, colind, val, x, lane);
        if (act && lane == 0) {
            const double ri = b[row] - ax;
            r[row] = ri;
            loc += ri * ri;
        }
    }
    const double bs = block_sum(loc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = bs;
    if (!last_block(&S->ticket1)) return;
    const double tot = reduce_parts_blk<BS>(part, gridDim.x, 1, 0, sh);
    if (threadIdx.x != 0) return;
    S->ticket1 = 0;
    if (S->bad || !(tot == tot)) { S->bad = 1; S->fin = 3; return; }
    S->rr_true = tot;
    S->last_upd = S->iters;
    if (tot <= S->threshold) { S->fin = 1; return; }
    if (S->iters >= S->max_iter) { S->fin = 2; return; }
    // six updates in a row that did not bring the best residual down by a
    // tenth: near the accuracy FP64 residuals can reach, the one-level
    // iteration may still get below a tolerance that this one circles
    S->stall = tot > 0.81 * S->rr_best ? S->stall + 1 : 0;
    S->rr_best = fmin(S->rr_best, tot);
    if (S->stall >= 6) { S->fin = 3; return; }
    S->fresh = S->rr_last > 0.0 && tot >= S->rr_last;
    S->rr_last = tot;
    // a recursion that agrees with the true residual may run twice as far (in
    // digits) before the next update, unless it has ever been far from it
    if (tot > 2.0 * S->rr) S->careful = 1;
    S->rrtrig = (!S->careful && tot < 1.003 * S->rr ? S->drop * S->drop : S->drop) * tot;
    S->rst = 1;
}

// without the FP64 matrix the iterated residual decides
__global__ void k_rl_iterated(CGScal* S) {
    if (!S->done || S->fin) return;
    S->rr_true = S->rr;
    S->fin = S->bad ? 3 : (S->done == 1 ? 1 : 2);
}

static void launch_rl_residual(isl_ctx* c, unsigned grid, cudaStream_t st, const double* x, double* r, CGScal* S) {
    const int n = (int)c->neq;
    const int *rp = c->drowptr.p, *ci = c->dcolind.p;
    const double *v = c->dval64.p, *b = c->drhs.p;
    double* part = c->dpart.p;
    switch (c->spmv_lpr64) {
        case 2: k_rl_residual<2><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, S, part); break;
        case 4: k_rl_residual<4><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, S, part); break;
        case 8: k_rl_residual<8><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, S, part); break;
        case 16: k_rl_residual<16><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, S, part); break;
        default: k_rl_residual<32><<<grid, BS, 0, st>>>(n, rp, ci, v, x, b, r, S, part); break;
    }
}

// slots in flight of the scalar two-level product: from the tuning cache, or
// timed (the first within 2 % of the fastest in a fixed order)
static int pz_kind(isl_ctx* c, const CzSpmv& m) {
    if (c->neq < 20000) return 108;
    const int cand[3] = {108, 104, 102};
    int cached = 0, best = 108;
    // (a key of its own: the one-level solve's kinds of these numbers are other kernels)
    if (tune_lookup(c, "spmv32_cz", &cached) && std::find(cand, cand + 3, cached) != cand + 3) return cached;
    float ms_of[3], bestms = 1e30f;
    cudaMemsetAsync(m.S, 0, sizeof(CGScal), c->stream);
    c->launches += 33;
    for (int k = 0; k < 3; ++k) {
        launch_coarse_spmv(c, cand[k], c->stream, m);
        cudaEventRecord(c->ev[2], c->stream);
        for (int r = 0; r < 10; ++r) launch_coarse_spmv(c, cand[k], c->stream, m);
        cudaEventRecord(c->ev[3], c->stream);
        cudaEventSynchronize(c->ev[3]);
        cudaEventElapsedTime(&ms_of[k], c->ev[2], c->ev[3]);
        bestms = std::min(bestms, ms_of[k]);
    }
    for (int k = 2; k >= 0; --k)
        if (ms_of[k] <= 1.02f * bestms) best = cand[k];
    tune_store(c, "spmv32_cz", best);
    return best;
}

// the one-launch form for small systems
static int solve_two_level_cluster(isl_ctx* c, int nc, bool grid, double tol, int64_t max_iter, int64_t* iters,
                                   double* rel, bool* ran) {
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq, na = (size_t)nc * c->cz.nrow;
    double* x64 = c->w64.p;
    float *V = c->w32.p, *d32 = nc == 3 ? c->dbinv.p : V + 3 * na;
    int rc = coarse_numeric(c, true, d32);
    if (rc != ISL_OK) return rc;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dscal.p, 0, sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, launch_coarse_cluster(c, grid, st, V, d32, x64, tol, c->have64 ? c->ru_drop2 : 0.0,
                                            (int)std::min<int64_t>(max_iter, INT32_MAX - 1)));
    c->launches += 1;
    rc = read_scal(c);
    if (rc != ISL_OK) return rc;
    const CGScal& h = *c->hscal;
    if (h.fault) ISL_FAIL(c, ISL_ERR_TIMEOUT, "two-level CG: a grid barrier timed out");
    if (h.fin != 1) return ISL_OK;
    *ran = true;
    *iters = h.iters;
    *rel = h.rhsNorm2 > 0 ? std::sqrt(h.rr_true / h.rhsNorm2) : 0.0;
    k_copy64<<<vec_grid(c), BS, 0, st>>>((int)n, x64, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}

// *ran = false: no usable coarse space, or the iteration broke down, stagnated
// or met its limit; the caller solves one-level, so that a solve that does not
// converge here ends as it does there
static int solve_two_level(isl_ctx* c, int nc, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* ran) {
    *ran = false;
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq;
    const int64_t rows = nc == 3 ? c->nbr : c->neq;
    const size_t na = (size_t)nc * rows;
    int rc = ISL_OK;
    if (nc == 3) {
        rc = ensure_bsr(c);
        if (rc != ISL_OK) return rc;
    }
    // One launch for the whole solve: a 16-CTA cluster for the smallest
    // systems (a cluster barrier costs less than a grid barrier), a
    // cooperative grid with one CTA per SM above (its shared memory holds
    // matrices of up to about 30 MB), up to the sizes where the one-level solve
    // leaves its one-launch kernels.  us per iteration, cluster / grid / three
    // graph launches, reliable updates included: 35k entries 9.5 / 11.3 / 28.7, 150k
    // 9.7 / 12.4 / -, 190k 15.1 / 12.7 / 33, 1.9M - / 13.3 / 22.5, 6.9M - / 26.3 /
    // 29.3 (the double-float sums since then: 0.2 to 0.7 more in one launch); in FP32
    // alone 35k 6.8 / - / 18.1, 146k 10.1 / - / 19.6, 187k - / 9.5 / 18.7, 1.9M - /
    // 11.7 / 20.9, 6.6M - / 24.7 / 25.9.  A context that shares the GPU with others
    // (side_by_side) takes the cluster, 16 SMs, or the graph.
    const int64_t ent = nc == 3 ? 9 * c->nblk : c->nnz;
    const bool one = c->use_persist == 1;
    if ((one || c->side_by_side) && rows <= (nc == 3 ? PERSIST_MAX_NBR : CLUSTER_MAX_N)) {
        for (int grid = one && ent > CZ_CLUSTER_ENTRIES; grid < (one ? 2 : 1); ++grid) {
            const int ncta = grid ? c->sm_count : cluster_ctas(c);
            if (ncta <= 0) continue;
            rc = coarse_plan(c, nc, rows, ncta);
            if (rc != ISL_OK || !c->cz.ok) return rc;
            const int fit = coarse_cluster_fits(c, grid != 0);
            if (grid ? fit > 0 : fit == 2) return solve_two_level_cluster(c, nc, grid != 0, tol, max_iter, iters, rel, ran);
        }
    }
    if (rows < (nc == 3 ? CZ_MIN_NODES : CZ_MIN_EQ)) return ISL_OK;
    rc = coarse_plan(c, nc, rows, 0);
    if (rc != ISL_OK || !c->cz.ok) return rc;
    const bool exact64 = c->have64;
    CGScal* S = c->dscal.p;
    double* W = c->w64.p;
    double *x64 = W, *r64 = W + n;
    float* V = c->w32.p;
    float *x32 = V, *r32 = V + na, *p32 = V + 2 * na, *q32 = V + 3 * na;
    float *z32 = nc == 3 ? V + 4 * na : V + 5 * na, *p32b = nc == 3 ? V + 5 * na : nullptr;
    float* d32 = nc == 3 ? c->dbinv.p : V + 4 * na;
    const unsigned grid = vec_grid(c);
    int kind;
    if (nc == 3) {
        if (!c->bspmv_lpb && c->nslot <= c->nblk + c->nblk / 10) {
            c->bspmv_lpb = 7;  // little padding: the batched sliced-ELL product, the autotune's first choice, without timing it
        } else if (!c->bspmv_lpb) {
            ISL_CHECK_CUDA(c, cudaMemsetAsync(p32, 0, na * 4, st));
            c->bspmv_lpb = autotune_lpb(c, p32, q32, S, c->dpart.p);
        }
        kind = c->nbr < 8000 ? 7 : c->bspmv_lpb;
        // below about a thousand slices the split product is the faster one
        // (solve at 9,261 nodes 3.48 ms against 4.06, at 31,744 4.45 against
        // 5.21; at 270,400 nodes 21.4 against 18.5)
        if (c->fuse_dir && c->nslice <= 1024) kind = 9;
    } else {
        kind = 108;
    }
    if (exact64 && !c->spmv_lpr64)
        c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, c->drhs.p, W + 3 * n, S, c->dpart.p);
    rc = coarse_numeric(c, false, d32);
    if (rc != ISL_OK) return rc;
    CzSpmv m = {};
    if (nc == 1) {
        rc = coarse_spmv_plan(c);
        if (rc != ISL_OK) return rc;
        m = {c->cz.bnd.p, c->cz.soff.p, c->cz.val.p, p32, q32, S, c->dpart.p, (int)rows};
        // (a CSR kind set through ISL_OPT_SPMV32_KIND is the one-level solve's)
        if (c->spmv32_forced >= 100) {
            c->cz.spmv_kind = c->spmv32_forced;
        } else if (!c->cz.spmv_kind) {
            ISL_CHECK_CUDA(c, cudaMemsetAsync(p32, 0, na * 4, st));
            c->cz.spmv_kind = pz_kind(c, m);
        }
        kind = c->cz.spmv_kind;
        c->spmv32_used = c->spmv32_forced ? c->spmv32_forced : kind;
    }
    const bool fused = nc == 3 && c->fuse_dir && (kind == 9 || bspmv_dir_kind(kind));
    CzIter a = {};
    coarse_args(c, a);
    a.x = x32; a.r = r32; a.z = z32;
    a.p1 = p32; a.p2 = fused ? p32b : nullptr; a.pz = p32;
    a.q = q32; a.dinv = nc == 3 ? c->cz.binv.p : d32; a.nrow = (int)rows;
    a.b64 = c->drhs.p;
    a.aeq = nc == 1 ? c->cz.perm.p : c->bpad ? c->dbaeq.p : nullptr;
    a.S = S; a.part = c->dpart.p;
    a.tol = tol; a.drop = exact64 ? c->ru_drop2 : 0.0;
    a.max_iter = (int)std::min<int64_t>(max_iter, INT32_MAX - 1);
    a.max_gap = coarse_gap(a.max_iter);
    ISL_CHECK_CUDA(c, cudaMemsetAsync(S, 0, 2 * sizeof(CGScal), st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(x64, 0, n * 8, st));
    launch_coarse(c, st, a, CZ_INIT);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 2;
    const int per_chunk = CZ_CHUNK * (fused ? 3 : 4) + (exact64 ? 4 : 2);
    // the captured iterations are kept while every argument stays the same
    // (the tolerance and the limits travel in the scalar record)
    a.b64 = r64;
    a.tol = a.drop = 0.0;
    a.max_iter = a.max_gap = 0;
    auto u = [](const void* p) { return (uint64_t)(uintptr_t)p; };
    std::vector<uint64_t> key = {(uint64_t)nc, (uint64_t)kind, (uint64_t)fused, (uint64_t)exact64, (uint64_t)rows, (uint64_t)n,
                                 (uint64_t)c->cz.nagg, (uint64_t)c->cz.ndp, (uint64_t)c->spmv_lpr64,
                                 (uint64_t)(c->use_scol16 && (nc == 3 ? c->scol16 : c->cz.short_cols)), (uint64_t)c->pattern_serial,
                                 u(a.lnode), u(a.sofs), u(a.dsub), u(a.ainv), u(a.rc), u(V), u(W), u(a.dinv), u(a.aeq), u(S),
                                 u(a.part), u(c->dsval.p), u(c->dbval.p), u(c->cz.val.p), u(c->dval32.p), u(c->dval64.p),
                                 u(c->drhs.p), u(c->drowptr.p), u(c->dcolind.p), u(c->dscol.p), u(c->dscol16.p), u(m.bnd), (uint64_t)c->cz.spmv_ncta,
                                 u(m.soff), u(c->cz.col.p), u(c->cz.col16.p)};
    if (!c->cz_exec || key != c->cz_key) {
        if (c->cz_exec) { cudaGraphExecDestroy(c->cz_exec); c->cz_exec = nullptr; }
        cudaGraph_t graph;
        ISL_CHECK_CUDA(c, cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        for (int k = 0; k < CZ_CHUNK; ++k) {
            if (fused) {
                launch_bspmv_dir(kind, st, c, z32, p32, p32b, q32, S, c->dpart.p);
            } else {
                launch_coarse_dir(c, st, (int)na, z32, p32, S);
                if (nc == 3) launch_bspmv(kind, grid, st, c, p32, q32, S, c->dpart.p);
                else launch_coarse_spmv(c, kind, st, m);
            }
            launch_coarse(c, st, a, CZ_UPDATE);
        }
        k_rl_fold<<<grid, BS, 0, st>>>((int)na, a.aeq, x32, x64, S);
        if (exact64) {
            launch_rl_residual(c, grid, st, x64, r64, S);
            launch_coarse(c, st, a, CZ_RESTART);
        } else {
            k_rl_iterated<<<1, 1, 0, st>>>(S);
        }
        ISL_CHECK_CUDA(c, cudaStreamEndCapture(st, &graph));
        cudaError_t e = cudaGraphInstantiate(&c->cz_exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) c->cz_exec = nullptr;
        ISL_CHECK_CUDA(c, e);
        c->cz_key = key;
    }
    for (auto& ev : c->cz_ev)
        if (!ev) ISL_CHECK_CUDA(c, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    // one graph in flight beyond the one whose record is being read
    const int64_t max_replays = (int64_t)std::min<int64_t>(max_iter, INT32_MAX - 1) + 64;
    int64_t k = 0;
    for (;; ++k) {
        if (k > max_replays) ISL_FAIL(c, ISL_ERR_TIMEOUT, "mixed CG made no progress");
        ISL_CHECK_CUDA(c, cudaGraphLaunch(c->cz_exec, st));
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->hscal + (k & 1), S, sizeof(CGScal), cudaMemcpyDeviceToHost, st));
        ISL_CHECK_CUDA(c, cudaEventRecord(c->cz_ev[k & 1], st));
        c->launches += per_chunk;
        if (k == 0) continue;
        ISL_CHECK_CUDA(c, cudaEventSynchronize(c->cz_ev[(k - 1) & 1]));
        if (c->hscal[(k - 1) & 1].fin) break;
    }
    const CGScal h = c->hscal[(k - 1) & 1];
    if (h.fin != 1) return ISL_OK;  // *ran stays false
    *ran = true;
    *iters = h.iters;
    *rel = h.rhsNorm2 > 0 ? std::sqrt(h.rr_true / h.rhsNorm2) : 0.0;
    k_copy64<<<grid, BS, 0, st>>>((int)n, x64, c->dsol.p);
    c->launches += 1;
    return ISL_OK;
}

int solve_device(isl_ctx* c, int method, double tol, int64_t max_iter, int64_t* iters, double* relres) {
    int rc = ensure_work(c);
    if (rc != ISL_OK) return rc;
    // every FP32 path but the node-blocked one reads the scalar FP32 CSR values
    if (method == ISL_SOLVE_CG_FP32_IR && !(c->blocked && c->use_block && (c->have64 || c->have32) && c->ninst == 1 &&
                                            !c->force_batched)) {
        rc = ensure_val32(c);
        if (rc != ISL_OK) return rc;
    }
    cudaStream_t st = c->stream;
    if (max_iter <= 0) max_iter = 2 * (int64_t)c->neq;
    if (c->timing) cudaEventRecord(c->ev[0], st);
    int64_t it = 0;
    double rel = 0.0;
    bool nc = false;
    if (c->ninst > 1 || (c->force_batched && method != ISL_SOLVE_BICGSTAB)) {
        rc = solve_batched(c, method, tol, max_iter, &it, &rel);
        nc = (rc == ISL_ERR_NOT_CONVERGED);
        if (rc == ISL_ERR_NOT_CONVERGED) rc = ISL_OK;
    } else if (method == ISL_SOLVE_BICGSTAB || method == ISL_SOLVE_CG_FP64) {
        const bool bicg = method == ISL_SOLVE_BICGSTAB;
        bool ran = false;
        if (!bicg || !c->bicg_forced) rc = solve_onelaunch(c, bicg, tol, max_iter, &it, &rel, &nc, &ran);
        if (rc == ISL_OK && ran && bicg && !c->bicg_lpr) c->bicg_lpr = 8;  // (reported for the one launch; the graph path still tunes)
        if (rc == ISL_OK && !ran)
            rc = bicg ? solve_bicgstab(c, tol, max_iter, &it, &rel, &nc) : solve_fp64(c, tol, max_iter, &it, &rel, &nc);
    }
    else {
        const bool b3 = c->blocked && c->use_block && (c->have64 || c->have32);
        bool ran = false;
        if (c->use_coarse && c->use_persist != 2 && (b3 ? c->nbr >= CZ_MIN_NODES_ONE : (int64_t)c->neq >= CZ_MIN_EQ)) {
            // a healthy two-level solve takes far fewer iterations than this
            const int64_t limit = std::min(max_iter, std::max<int64_t>(1000, (int64_t)c->neq / 4));
            rc = solve_two_level(c, b3 ? 3 : 1, tol, limit, &it, &rel, &ran);
            if (rc == ISL_ERR_NOMEM) {  // no room for the coarse space: one-level
                coarse_drop(c);
                rc = ISL_OK;
            }
        }
        if (rc == ISL_OK && !ran)
            rc = b3 ? solve_mixed_b3(c, tol, max_iter, &it, &rel, &nc) : solve_mixed(c, tol, max_iter, &it, &rel, &nc);
    }
    if (rc != ISL_OK) return rc;
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    if (c->timing) {
        cudaEventRecord(c->ev[1], st);
        cudaEventSynchronize(c->ev[1]);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
        c->tms[ISL_T_SOLVE] += ms;
        c->tcount[ISL_T_SOLVE]++;
    }
    c->solved = true;
    if (iters) *iters = it;
    if (relres) *relres = rel;
    if (nc) ISL_FAIL(c, ISL_ERR_NOT_CONVERGED, "solver did not reach the tolerance");
    return ISL_OK;
}

__global__ void k_distribute(int64_t ndc, const int32_t* __restrict__ eq, const uint8_t* __restrict__ status,
                             const double* __restrict__ cval, const double* __restrict__ x, double* __restrict__ u, int add) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < ndc; k += (int64_t)gridDim.x * blockDim.x) {
        if (status[k] == 0) u[k] = add ? u[k] + x[eq[k]] : x[eq[k]];
        else u[k] = cval[k];
    }
}

int distribute_device(isl_ctx* c, int add) {
    const int64_t ndc = c->ndofobj * c->ncomp;
    k_distribute<<<vec_grid(c), BS, 0, c->stream>>>(ndc, c->deq.p, c->dstatus.p, c->dcval.p, c->dsol.p, c->du.p, add);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 1;
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(c->stream));
    return ISL_OK;
}

int time_spmv(isl_ctx* c, int precision, int nrep, double* ms) {
    if (c->ninst > 1 || c->force_batched) return time_spmv_batched(c, precision, std::abs(nrep), ms);
    const bool warm = nrep > 0;  // one untimed launch first
    nrep = std::abs(nrep);
    int rc = ensure_work(c);
    if (rc != ISL_OK) return rc;
    const size_t n = (size_t)c->neq;
    CGScal* S = c->dscal.p;
    cudaStream_t st = c->stream;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(S, 0, sizeof(CGScal), st));
    if (precision == ISL_PREC_FP32 && c->blocked && c->use_block) {
        if (!c->have32) ISL_FAIL(c, ISL_ERR_ARG, "no FP32 matrix");
        return time_bspmv(c, warm ? nrep : -nrep, ms);
    }
    if (precision == ISL_PREC_FP32) {
        if (!c->have32) ISL_FAIL(c, ISL_ERR_ARG, "no FP32 matrix");
        rc = ensure_val32(c);
        if (rc != ISL_OK) return rc;
        float* V = c->w32.p;
        ISL_CHECK_CUDA(c, cudaMemsetAsync(V + 2 * n, 0, n * 4, st));
        const CzPlan& z = c->cz;
        const bool csr = c->spmv32_forced > 0 && c->spmv32_forced < 100;  // (set: the one-level product)
        if (z.spmv_kind && !csr && c->use_coarse && c->use_persist != 2 && z.ok && z.nc == 1 && z.serial == c->pattern_serial && z.sell_built &&
            z.sell_serial == c->asm_serial && z.bnd_serial == z.serial) {  // the product of the two-level solve that ran
            const CzSpmv m = {z.bnd.p, z.soff.p, z.val.p, V + 2 * n, V + 3 * n, S, c->dpart.p, (int)n};
            if (warm) launch_coarse_spmv(c, z.spmv_kind, st, m);
            cudaEventRecord(c->ev[2], st);
            for (int r = 0; r < nrep; ++r) launch_coarse_spmv(c, z.spmv_kind, st, m);
            cudaEventRecord(c->ev[3], st);
            ISL_CHECK_CUDA(c, cudaEventSynchronize(c->ev[3]));
            float t = 0.f;
            cudaEventElapsedTime(&t, c->ev[2], c->ev[3]);
            *ms = (double)t / nrep;
            c->launches += nrep + (warm ? 1 : 0);
            return ISL_OK;
        }
        rc = ensure_ssell(c);
        if (rc != ISL_OK) return rc;
        if (!c->spmv_lpr32) c->spmv_lpr32 = autotune_spmv32(c, V + 2 * n, V + 3 * n, S, c->dpart.p);
        c->spmv32_used = c->spmv_lpr32;
        if (warm) launch_spmv32(c, c->spmv_lpr32, vec_grid(c), st, V + 2 * n, V + 3 * n, S, c->dpart.p);
        cudaEventRecord(c->ev[2], st);
        for (int r = 0; r < nrep; ++r) launch_spmv32(c, c->spmv_lpr32, vec_grid(c), st, V + 2 * n, V + 3 * n, S, c->dpart.p);
        cudaEventRecord(c->ev[3], st);
    } else {
        if (!c->have64) ISL_FAIL(c, ISL_ERR_ARG, "no FP64 matrix");
        double* W = c->w64.p;
        ISL_CHECK_CUDA(c, cudaMemsetAsync(W + 2 * n, 0, n * 8, st));
        if (!c->spmv_lpr64) c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, W + 2 * n, W + 3 * n, S, c->dpart.p);
        if (warm)
            launch_spmv<double, double>(c->spmv_lpr64, vec_grid(c), st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, W + 2 * n, W + 3 * n, S, c->dpart.p);
        cudaEventRecord(c->ev[2], st);
        for (int r = 0; r < nrep; ++r)
            launch_spmv<double, double>(c->spmv_lpr64, vec_grid(c), st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, W + 2 * n, W + 3 * n, S, c->dpart.p);
        cudaEventRecord(c->ev[3], st);
    }
    c->launches += nrep + (warm ? 1 : 0);
    ISL_CHECK_CUDA(c, cudaEventSynchronize(c->ev[3]));
    float t = 0.f;
    cudaEventElapsedTime(&t, c->ev[2], c->ev[3]);
    *ms = t / nrep;
    ISL_CHECK_CUDA(c, cudaGetLastError());
    return ISL_OK;
}


// Warm per-kernel timing of one CG iteration's kernels (CUDA events around nrep
// back-to-back launches each).  ms[0] block SpMV (autotuned kind), ms[1]
// block-Jacobi update, ms[2] block-Jacobi direction, ms[3] FP64 CSR SpMV,
// ms[4] FP64 update, ms[5] FP64 direction, ms[6] FP64 residual, ms[7] = the
// chosen block SpMV kind (or -1 when the pattern is not node-blocked).
int time_kernels(isl_ctx* c, int nrep, double* ms) {
    int rc = ensure_work(c);
    if (rc != ISL_OK) return rc;
    cudaStream_t st = c->stream;
    const size_t n = (size_t)c->neq;
    const unsigned grid = vec_grid(c);
    CGScal h;
    memset(&h, 0, sizeof(h));
    h.absNew = 1.0; h.absOld = 1.0; h.alpha = 1e-6; h.beta = 0.5; h.threshold = -1.0; h.rrtrig = -1.0;
    auto reset = [&]() { return cudaMemcpyAsync(c->dscal.p, &h, sizeof(h), cudaMemcpyHostToDevice, st); };
    auto timeit = [&](auto&& launch) -> double {
        reset();
        launch();
        cudaEventRecord(c->ev[2], st);
        for (int r = 0; r < nrep; ++r) launch();
        cudaEventRecord(c->ev[3], st);
        cudaEventSynchronize(c->ev[3]);
        float t = 0.f;
        cudaEventElapsedTime(&t, c->ev[2], c->ev[3]);
        return t / nrep;
    };
    const int mi = INT32_MAX - 1;
    for (int k = 0; k < 8; ++k) ms[k] = -1.0;
    if (c->blocked && c->have32) {
        rc = ensure_bsr(c);
        if (rc != ISL_OK) return rc;
        float* V = c->w32.p;
        const size_t na = (size_t)3 * c->nbr;  // the block space (padded blocks included)
        float *x = V, *r = V + na, *p = V + 2 * na, *q = V + 3 * na;
        k_fill<<<grid, BS, 0, st>>>((int64_t)(4 * na), V, 1.0f);
        if (!c->bspmv_lpb) c->bspmv_lpb = autotune_lpb(c, p, q, c->dscal.p, c->dpart.p);
        const int nbr = (int)c->nbr;
        const unsigned nbd = (unsigned)std::max<long long>(1, (3LL * nbr + NBS - 1) / NBS);
        if (c->fuse_dir && bspmv_dir_kind(c->bspmv_lpb)) {
            // what the mixed solve launches: the product with the direction
            // update folded in, and the update that stores z
            float *z = V + 4 * na, *pb = V + 5 * na;
            k_fill<<<grid, BS, 0, st>>>((int64_t)(2 * na), z, 1.0f);
            ms[0] = timeit([&] { launch_bspmv_dir(c->bspmv_lpb, st, c, z, p, pb, q, c->dscal.p, c->dpart.p); });
            const int uk = c->bupd_kind[1] ? c->bupd_kind[1] : 1;
            ms[1] = timeit([&] { launch_update(c, uk, true, st, x, r, p, pb, q, z, c->dscal.p, mi); });
        } else {
            ms[0] = timeit([&] { launch_bspmv(c->bspmv_lpb, grid, st, c, p, q, c->dscal.p, c->dpart.p); });
            const int uk = c->bupd_kind[0] ? c->bupd_kind[0] : 1;
            ms[1] = timeit([&] { launch_update(c, uk, false, st, x, r, p, p, q, nullptr, c->dscal.p, mi); });
            ms[2] = timeit([&] { k_cg_dir_b3<<<nbd, NBS, 0, st>>>(nbr, r, c->dbinv.p, p, c->dscal.p); });
        }
        ms[7] = c->bspmv_lpb;
    }
    if (c->have64) {
        double* W = c->w64.p;
        double *x = W, *r = W + n, *p = W + 2 * n, *q = W + 3 * n, *dinv = W + 4 * n, *r64 = W + 5 * n;
        k_fill64<<<grid, BS, 0, st>>>((int64_t)(6 * n), W, 1.0);
        if (!c->spmv_lpr64) c->spmv_lpr64 = autotune_lpr<double, double>(c, c->dval64.p, p, q, c->dscal.p, c->dpart.p);
        const int lpr = c->spmv_lpr64;
        double* dres = (double*)(c->dscal.p + 1);
        unsigned* ticket = &(c->dscal.p + 1)->ticket1;
        ms[3] = timeit([&] { launch_spmv<double, double>(lpr, grid, st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, p, q, c->dscal.p, c->dpart.p); });
        ms[4] = timeit([&] { k_cg_update<double><<<upd_grid(c, n), BS, 0, st>>>((int)n, x, r, p, q, dinv, c->dscal.p, c->dpart.p, mi); });
        const unsigned gdir = (unsigned)std::max<long long>(1, ((long long)n + BS - 1) / BS);
        ms[5] = timeit([&] { k_cg_dir<double><<<gdir, BS, 0, st>>>((int)n, r, dinv, p, c->dscal.p); });
        ms[6] = timeit([&] { launch_residual(lpr, grid, st, (int)n, c->drowptr.p, c->dcolind.p, c->dval64.p, x, c->drhs.p, r64, c->dpart.p, ticket, dres); });
    }
    c->launches += 7 * (nrep + 1);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    return ISL_OK;
}

}  // namespace isl

// ---------------------------------------------------------------------------
// isl_cg_solve_noalloc: the FP64 Jacobi CG above (same init, direction, SpMV
// and update kernels) on caller-owned device buffers, with its work vectors in
// a fixed device array instead of memory allocated per call.
//
// Scratch layout (doubles): the CG scalars (256 bytes), two partial sums per
// block of the largest grid, then r, p, q and the inverse diagonal, each
// ISL_NOALLOC_MAX_N long.  The iterate is the caller's x.
namespace {
constexpr int NA_MAX_N = ISL_NOALLOC_MAX_N;
constexpr int NA_MAX_BLOCKS = 4096;
constexpr int NA_MAX_DEVICES = 64;
constexpr size_t NA_PART_OFF = 32;
constexpr size_t NA_VEC_OFF = NA_PART_OFF + 2 * (size_t)NA_MAX_BLOCKS;
constexpr size_t NA_WORDS = NA_VEC_OFF + 4 * (size_t)NA_MAX_N;
static_assert(sizeof(isl::CGScal) <= NA_PART_OFF * sizeof(double), "CG scalars exceed their scratch slot");
static_assert(NA_VEC_OFF % 32 == 0, "vectors start on 256-byte boundaries");
}  // namespace

static __device__ __align__(256) double g_noalloc_scratch[NA_WORDS];

namespace isl {
namespace {

// diagonal of a caller CSR row (first stored entry with col == row); rows
// without a nonzero diagonal get 1, as the Jacobi preconditioner above does
__global__ void k_noalloc_dinv(int n, const int* __restrict__ rowptr, const int* __restrict__ colind,
                               const double* __restrict__ val, double* __restrict__ dinv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double d = 0.0;
        for (int k = rowptr[i]; k < rowptr[i + 1]; ++k)
            if (colind[k] == i) { d = val[k]; break; }
        dinv[i] = (d != 0.0) ? 1.0 / d : 1.0;
    }
}

struct NoallocDevice {
    double* base = nullptr;  // device address of g_noalloc_scratch on this device
    void* cuctx = nullptr;   // driver context the address belongs to
    int sms = 0;
};
std::mutex g_noalloc_mu;
NoallocDevice g_noalloc_dev[NA_MAX_DEVICES];

// cuCtxGetCurrent through the runtime's driver entry point (the library links
// only the runtime): the current context identifies a device's module
// instance, which changes when cudaDeviceReset destroys the primary context
typedef int (*CtxGetCurrentFn)(void**);
CtxGetCurrentFn noalloc_ctx_fn() {
    static CtxGetCurrentFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (CtxGetCurrentFn)f;
    }();
    return fn;
}

// once per device context, with that device current: the scratch array's
// address.  A reset device gets a new primary context and module instance,
// so the address is looked up again when the current context changes.
int noalloc_setup(int device, NoallocDevice* out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoallocDevice& e = g_noalloc_dev[device];
    void* cur = nullptr;
    CtxGetCurrentFn fn = noalloc_ctx_fn();
    if (!fn || fn(&cur) != 0) return ISL_ERR_CUDA;
    double* ptr = nullptr;
    if (!cur) {
        // no context current on this thread yet: the runtime call creates
        // (or binds) the device's primary context
        if (cudaGetSymbolAddress((void**)&ptr, g_noalloc_scratch) != cudaSuccess || !ptr) return ISL_ERR_CUDA;
        if (fn(&cur) != 0 || !cur) return ISL_ERR_CUDA;
    }
    if (!e.base || e.cuctx != cur) {
        if (!ptr && (cudaGetSymbolAddress((void**)&ptr, g_noalloc_scratch) != cudaSuccess || !ptr)) return ISL_ERR_CUDA;
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
            return ISL_ERR_CUDA;
        e.sms = sms;
        e.base = ptr;
        e.cuctx = cur;
    }
    *out = e;
    return ISL_OK;
}

int noalloc_cg(const NoallocDevice& dv, cudaStream_t st, int n, const int* rowptr, const int* colind, const double* val,
               const double* b, double* x, double tol, int64_t max_iter, int64_t* iters, double* rel_res) {
    CGScal* S = reinterpret_cast<CGScal*>(dv.base);
    double* part = dv.base + NA_PART_OFF;
    double* r = dv.base + NA_VEC_OFF;
    double *p = r + NA_MAX_N, *q = p + NA_MAX_N, *dinv = q + NA_MAX_N;
    // SpMV variant by the mean row length (lanes per row)
    int nnz = 0;
    if (cudaMemcpyAsync(&nnz, rowptr + n, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return ISL_ERR_CUDA;
    if (nnz < 0) return ISL_ERR_ARG;
    const double avg = (double)nnz / n;
    const int lpr = avg <= 6 ? 2 : avg <= 12 ? 4 : avg <= 24 ? 8 : avg <= 48 ? 16 : 32;
    const int mi = (int)std::min<int64_t>(max_iter <= 0 ? 2 * (int64_t)n : max_iter, INT32_MAX - 1);
    const unsigned gvec = (unsigned)std::min(8 * dv.sms, NA_MAX_BLOCKS);
    const unsigned gupd = (unsigned)std::max(1, std::min((n + BS - 1) / BS, 2 * dv.sms));
    const unsigned gdir = (unsigned)((n + BS - 1) / BS);
    // the scalars hold the reduction tickets, the counters and the done flag:
    // they must start at zero; every vector is written before it is read
    // iters / rel_res come from the last scalar record read back, on every
    // return after the solve started (zero before the first read)
    CGScal h{};
    auto report = [&](int rc) {
        if (iters) *iters = h.iters;
        if (rel_res) *rel_res = h.rhsNorm2 > 0 ? std::sqrt(h.rr / h.rhsNorm2) : 0.0;
        return rc;
    };
    if (cudaMemsetAsync(S, 0, sizeof(CGScal), st) != cudaSuccess) return report(ISL_ERR_CUDA);
    k_noalloc_dinv<<<gdir, BS, 0, st>>>(n, rowptr, colind, val, dinv);
    k_cg_init<double, double><<<gvec, BS, 0, st>>>(n, b, x, r, p, dinv, S, part, tol, 0.0);
    if (cudaGetLastError() != cudaSuccess) return report(ISL_ERR_CUDA);
    const int64_t max_rounds = (int64_t)mi / CHUNK + 3;
    for (int64_t round = 0;; ++round) {
        CGScal t;
        if (cudaMemcpyAsync(&t, S, sizeof(CGScal), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return report(ISL_ERR_CUDA);
        h = t;
        if (h.done) break;
        if (round > max_rounds) return report(ISL_ERR_TIMEOUT);
        for (int k = 0; k < CHUNK; ++k) {
            k_cg_dir<double><<<gdir, BS, 0, st>>>(n, r, dinv, p, S);
            launch_spmv<double, double>(lpr, gvec, st, n, rowptr, colind, val, p, q, S, part);
            k_cg_update<double><<<gupd, BS, 0, st>>>(n, x, r, p, q, dinv, S, part, mi);
        }
        if (cudaGetLastError() != cudaSuccess) return report(ISL_ERR_CUDA);
    }
    if (h.bad) return report(ISL_ERR_NAN);
    if (h.done == 2) return report(ISL_ERR_NOT_CONVERGED);
    return report(ISL_OK);
}

}  // namespace
}  // namespace isl

extern "C" int isl_cg_solve_noalloc(int device, void* stream, int n, const int32_t* rowptr, const int32_t* colind,
                                    const double* val, const double* b, double* x, double tol, int64_t max_iter,
                                    int64_t* iters, double* rel_res) {
    if (n < 0 || !(tol >= 0.0)) return ISL_ERR_ARG;
    if (n > ISL_NOALLOC_MAX_N) return ISL_ERR_CAPACITY;
    if (n == 0) {
        if (iters) *iters = 0;
        if (rel_res) *rel_res = 0.0;
        return ISL_OK;
    }
    if (!rowptr || !colind || !val || !b || !x) return ISL_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess) return ISL_ERR_CUDA;
    if (device < 0 || device >= ndev || device >= NA_MAX_DEVICES) return ISL_ERR_ARG;
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) return ISL_ERR_CUDA;
    if (prev != device && cudaSetDevice(device) != cudaSuccess) return ISL_ERR_CUDA;
    isl::NoallocDevice dv;
    int rc = isl::noalloc_setup(device, &dv);
    if (rc == ISL_OK)
        rc = isl::noalloc_cg(dv, (cudaStream_t)stream, n, rowptr, colind, val, b, x, tol, max_iter, iters, rel_res);
    if (prev != device) cudaSetDevice(prev);
    return rc;
}
