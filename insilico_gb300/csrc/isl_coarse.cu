// Two-level preconditioner of the mixed CG (single systems and the instances of a
// batch).
//
//   M^-1 = D0^-1 + sum_s P_s D_s^-1 P_s^T + P A_c^-1 P^T
//
// D0: the (block) diagonal, as in the one-level solve.  P: the field's rows
// are grouped into aggregates, the boxes of a quantile grid over the DOF
// objects' support points, each box split in two per direction into
// sub-aggregates s.  Every aggregate carries the smooth modes of its rows:
// the constant and the linear functions of a scalar equation, the six
// rigid-body modes of a 3-component node block.  D_s is the Galerkin block of
// one sub-aggregate, A_c = P^T A P the Galerkin matrix of all aggregates,
// inverted dense.
//
// Jacobi CG needs about as many iterations as the mesh has cells across
// (2,257 for 64^3 elasticity at 1e-10, 801 for 40^3 P2 tetrahedra); with the
// coarse space the count depends on the cells across one aggregate instead.
// Each term is symmetric positive (semi-)definite for any choice of boxes, so
// the boxes need no connectivity and the sum is a CG preconditioner on any
// mesh.
//
// Measured (solve with the numeric setup of the assembly, 1e-10): 64^3
// elasticity 144 -> 17.8 ms (194 iterations instead of 2,257; setup 1.3 ms),
// 20^3 13.6 -> 1.9 ms, 40^3 P2 tetrahedra 38.9 -> 8.9 ms, Q2 160^2 24.2 -> 5.1 ms.
//
// Cost per iteration beyond the one-level solve: the update kernel takes one
// CTA per aggregate and one warp per sub-aggregate, so the restriction and the
// sub-aggregate solve stay inside a warp; one more launch multiplies by the
// dense inverse (its rows for one aggregate per CTA) and prolongs into z.
//
// Determinism: the rows of a sub-aggregate are listed in a fixed order (ascending,
// scalar rows by their length first) and summed in it; the coarse entries between
// aggregates, which several threads add to, are summed in 64-bit fixed point.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include "isl_coarse.h"
#include "isl_device.cuh"

namespace isl {

namespace {

constexpr int TB = COARSE_TILE;   // tile of the dense inversion
constexpr int NBIN = 1024;        // bins per axis of the quantile cuts
constexpr int ROW_BITS = 29;      // lnode.w: row, and the constrained components of a padded node block above
constexpr float REG = 1e-5f;      // added to the unit diagonal of the scaled coarse matrices
constexpr int CZ_KEEP = 2;        // rows of a thread that k_cz_update and k_cz_coarse hold in registers
constexpr int FIX_BITS = 32;      // fixed point of the coarse entries: the bound of an entry is 2^32

__device__ inline int lrow(float4 l) { return __float_as_int(l.w) & ((1 << ROW_BITS) - 1); }
__device__ inline int lmask(float4 l) { return (int)((unsigned)__float_as_int(l.w) >> ROW_BITS); }

// modes of one row: NC = 1: 1, y0, y1 (, y2); NC = 3: translations, rotations
template <int NC, int M>
__device__ __forceinline__ void restrict_add(float (&rc)[M], const float (&r)[NC], const float4& y) {
    if constexpr (NC == 1) {
        rc[0] += r[0];
        rc[1] += r[0] * y.x;
        rc[2] += r[0] * y.y;
        if constexpr (M == 4) rc[3] += r[0] * y.z;
    } else {
        rc[0] += r[0]; rc[1] += r[1]; rc[2] += r[2];
        rc[3] += r[2] * y.y - r[1] * y.z;
        rc[4] += r[0] * y.z - r[2] * y.x;
        rc[5] += r[1] * y.x - r[0] * y.y;
    }
}
template <int NC, int M>
__device__ __forceinline__ void prolong(const float (&c)[M], const float4& y, float (&o)[NC]) {
    if constexpr (NC == 1) {
        o[0] = c[0] + c[1] * y.x + c[2] * y.y;
        if constexpr (M == 4) o[0] += c[3] * y.z;
    } else {
        o[0] = c[0] + c[4] * y.z - c[5] * y.y;
        o[1] = c[1] + c[5] * y.x - c[3] * y.z;
        o[2] = c[2] + c[3] * y.y - c[4] * y.x;
    }
}

// Sums of the (hi, lo) pairs part[i].xy and .zw, i < n, by warp 0 (at most a
// few hundred partials, one per aggregate): ten loads in flight per lane, one
// round trip for 320 blocks, and no block barrier.  Valid in warp 0.
__device__ __forceinline__ void reduce_parts2_df_warp(const float4* part, int n, df& s0, df& s1) {
    s0 = s1 = {0.f, 0.f};
    if (threadIdx.x >= 32) return;
    for (int base = 0; base < n; base += 320) {
        float4 v[10];
#pragma unroll
        for (int u = 0; u < 10; ++u) {
            const int i = base + u * 32 + (int)threadIdx.x;
            v[u] = i < n ? __ldcg(part + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 10; ++u) {
            s0 = df_add_acc(s0, df{v[u].x, v[u].y});
            s1 = df_add_acc(s1, df{v[u].z, v[u].w});
        }
    }
    s0 = warp_sum_df(s0);
    s1 = warp_sum_df(s1);
}

// ---------------------------------------------------------------------------
// Iteration kernels

template <int NC>
struct Row {
    float4 L;
    float x[NC], r[NC];
};

// One CTA per aggregate, WPS warps per sub-aggregate.
//   CZ_UPDATE : x += alpha p, r -= alpha q
//   CZ_INIT   : r = b, x = p = 0
//   CZ_RESTART: r = the FP64 residual (reliable update)
// then z = D0^-1 r + P_s D_s^-1 P_s^T r, the aggregate's entries of P^T r, and
// the sums r.r and r.z (without the coarse term, which k_cz_coarse adds).
template <int NC, int M, int NW, int WPS, int MODE>
__global__ void __launch_bounds__(NW * WPS * 32) k_cz_update(CzIter a) {
    CGScal* S = a.S;
    __shared__ double sh[64];
    __shared__ float src[NW * WPS][M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sl = w / WPS, sub = blockIdx.x * NW + sl;
    chain_next();
    const int t0 = a.sofs[sub] + (w % WPS) * 32 + lane, t1 = a.sofs[sub + 1];
    Row<NC> Rk[CZ_KEEP];
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + 32 * WPS * k < t1) Rk[k].L = __ldg(a.lnode + t0 + 32 * WPS * k);
    // row m of the sub-aggregate's inverse block, in lane m
    float Dm[M];
#pragma unroll
    for (int k = 0; k < M; ++k) Dm[k] = lane < M ? __ldg(a.dsub + (size_t)sub * (M * M) + M * lane + k) : 0.f;
    chain_wait();
    if (MODE == CZ_UPDATE && S->done) return;
    if (MODE == CZ_RESTART && !S->rst) return;
    const float* p = (a.p2 && !(S->iters & 1)) ? a.p2 : a.p1;
    const float alpha = MODE == CZ_UPDATE ? (float)S->alpha : 0.f;
    float rc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) rc[m] = 0.f;
    typename std::conditional<MODE == CZ_UPDATE, float, double>::type rr = 0, rz = 0;  // (FP64 where it costs nothing)
    double bb = 0.0;
    // loads of a row, then (in row_step) its stores: the rows held in registers load together
    auto row_load = [&](Row<NC>& R) {
        const size_t d = (size_t)NC * lrow(R.L);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (MODE == CZ_UPDATE) {
                R.x[c] = a.x[d + c] + alpha * p[d + c];
                R.r[c] = a.r[d + c] - alpha * a.q[d + c];
            } else {
                const int e = a.aeq ? a.aeq[d + c] : (int)(d + c);
                const double v = e >= 0 ? a.b64[e] : 0.0;
                R.r[c] = (float)v;
                if (MODE == CZ_INIT) bb += v * v;
            }
        }
    };
    auto row_step = [&](int t, const Row<NC>& R, float (&zv)[NC]) {
        const size_t d = (size_t)NC * lrow(R.L);
        float bi[NC * NC];
#pragma unroll
        for (int k = 0; k < NC * NC; ++k) bi[k] = __ldg(a.dinv + (size_t)k * a.nrow + t);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (MODE == CZ_UPDATE) a.x[d + c] = R.x[c];
            if (MODE == CZ_INIT) a.x[d + c] = a.pz[d + c] = 0.f;
            a.r[d + c] = R.r[c];
            zv[c] = 0.f;
#pragma unroll
            for (int k = 0; k < NC; ++k) zv[c] += bi[NC * c + k] * R.r[k];
            rr += (decltype(rr))R.r[c] * R.r[c];
            rz += (decltype(rz))R.r[c] * zv[c];
        }
        restrict_add<NC, M>(rc, R.r, R.L);
    };
    // the first rows of a thread stay in registers with their part of z
    float zk[CZ_KEEP][NC];
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + 32 * WPS * k < t1) row_load(Rk[k]);
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + 32 * WPS * k < t1) row_step(t0 + 32 * WPS * k, Rk[k], zk[k]);
#pragma unroll 1
    for (int t = t0 + 32 * WPS * CZ_KEEP; t < t1; t += 32 * WPS) {
        Row<NC> R;
        float zv[NC];
        R.L = __ldg(a.lnode + t);
        row_load(R);
        row_step(t, R, zv);
#pragma unroll
        for (int c = 0; c < NC; ++c) a.z[(size_t)NC * lrow(R.L) + c] = zv[c];
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rc[m] += __shfl_xor_sync(0xffffffffu, rc[m], o);
    if (lane == 0) {
#pragma unroll
        for (int m = 0; m < M; ++m) src[w][m] = rc[m];
    }
    __syncthreads();
    if (WPS > 1) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
            rc[m] = 0.f;
#pragma unroll
            for (int k = 0; k < WPS; ++k) rc[m] += src[sl * WPS + k][m];
        }
    }
    float z1[M], zm = 0.f, rz1 = 0.f;
#pragma unroll
    for (int k = 0; k < M; ++k) zm += Dm[k] * rc[k];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        z1[m] = __shfl_sync(0xffffffffu, zm, m);
        rz1 += rc[m] * z1[m];
    }
    if (w % WPS == 0 && lane == 0) rz += rz1;
    auto add_sub = [&](const float4& L, const float (&zv)[NC]) {
        const size_t d = (size_t)NC * lrow(L);
        float o[NC];
        prolong<NC, M>(z1, L, o);
        const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
        for (int c = 0; c < NC; ++c) a.z[d + c] = (mk >> c) & 1 ? zv[c] : zv[c] + o[c];
    };
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + 32 * WPS * k < t1) add_sub(Rk[k].L, zk[k]);
#pragma unroll 1
    for (int t = t0 + 32 * WPS * CZ_KEEP; t < t1; t += 32 * WPS) {  // each thread adds to the entries of z it wrote
        const float4 L = __ldg(a.lnode + t);
        float zv[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) zv[c] = a.z[(size_t)NC * lrow(L) + c];
        add_sub(L, zv);
    }
    if (threadIdx.x < M) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < NW * WPS; ++k) s += src[k][threadIdx.x];
        a.rc[(size_t)blockIdx.x * M + threadIdx.x] = s;
    }
    double trr;
    df trz;
    if constexpr (MODE != CZ_UPDATE) {
        const double b1 = block_sum(MODE == CZ_INIT ? bb : rr, sh);
        const double b2 = block_sum(rz, sh);
        if (threadIdx.x == 0) { a.part[2 * blockIdx.x] = b1; a.part[2 * blockIdx.x + 1] = b2; }
        if (!last_block(&S->ticket2)) return;
        double t;
        reduce_parts2(a.part, gridDim.x, sh, trr, t);
        trz = df_from_double(t);
    } else {
        df b1, b2;
        block_sum_df2(rr, rz, reinterpret_cast<float*>(sh), b1, b2);
        if (threadIdx.x == 0) reinterpret_cast<float4*>(a.part)[blockIdx.x] = make_float4(b1.hi, b1.lo, b2.hi, b2.lo);
        if (!last_block(&S->ticket2)) return;
        df t;
        reduce_parts2_df_warp(reinterpret_cast<const float4*>(a.part), gridDim.x, t, trz);
        trr = df_value(t);
    }
    if (threadIdx.x != 0) return;
    S->rr = trr;
    S->rzloc = make_float2(trz.hi, trz.lo);
    S->ticket2 = 0;
    if (MODE == CZ_UPDATE) {
        S->iters += 1;
        S->absOld = S->absNew;
        S->rz_old = S->rz_new;
        if (!(trr == trr) || !(trz.hi == trz.hi)) { S->bad = 1; S->done = 1; }
        else if (trr < S->threshold) S->done = 1;
        else if (trr < S->rrtrig || (S->drop > 0.0 && trr > 1e8 * S->rr_true)) S->done = 3;  // dropped enough, or diverging
        else if (S->iters >= S->max_iter) S->done = 2;
        else if (S->drop > 0.0 && S->iters - S->last_upd >= S->max_gap) { S->bad = 1; S->done = 1; }
    } else if (MODE == CZ_INIT) {
        S->rhsNorm2 = trr;
        S->rr_true = trr;
        S->rr_last = 0.0;
        S->rr_best = trr;
        S->stall = 0;
        S->careful = 0;
        S->threshold = a.tol * a.tol * trr;
        S->rrtrig = a.drop * trr;
        S->drop = a.drop;
        S->max_iter = a.max_iter;
        S->max_gap = a.max_gap;
        S->last_upd = 0;
        S->iters = 0;
        S->beta = 0.0;
        S->rst = 0;
        S->bad = !(trr == trr);
        S->done = (trr == 0.0 || trr < S->threshold || S->bad) ? 1 : 0;
        S->fin = S->bad ? 3 : (trr == 0.0 ? 1 : 0);
        S->ticket1 = 0;
    }
}

// z += P A_c^-1 P^T r: one CTA per aggregate computes its M rows of the dense
// inverse times P^T r (PR warps per row) and prolongs them to its own rows of
// z; the last block adds the coarse term of r.z and forms beta.  The inverse
// (13 MB at 300 aggregates of node blocks) is read once per iteration.
template <int NC, int M, int NW, int WPS, int MODE>
__global__ void __launch_bounds__(NW * WPS * 32) k_cz_coarse(CzIter a) {
    constexpr int TW = NW * WPS, PR = TW >= M ? TW / M : 1;
    CGScal* S = a.S;
    __shared__ float zs[PR][M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n4 = a.ndp / 4;
    const float4* rc4 = reinterpret_cast<const float4*>(a.rc);
    chain_next();
    const int t0 = a.sofs[blockIdx.x * NW] + (int)threadIdx.x, t1 = a.sofs[(blockIdx.x + 1) * NW];
    float4 Lk[CZ_KEEP];
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + TW * 32 * k < t1) Lk[k] = __ldg(a.lnode + t0 + TW * 32 * k);
    // the dense rows of the aggregate into the L2 (the product streams the matrix through it)
    for (int k = threadIdx.x; k < M * a.ndp / 32; k += TW * 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.ainv + (size_t)blockIdx.x * M * a.ndp + 32 * k));
    chain_wait();
    if (MODE != CZ_RESTART && S->done) return;
    if (MODE == CZ_RESTART && !S->rst) return;
    // z of the first rows of a thread is on its way while the dense rows are multiplied
    float zk[CZ_KEEP][NC];
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + TW * 32 * k < t1) {
#pragma unroll
            for (int c = 0; c < NC; ++c) zk[k][c] = a.z[(size_t)NC * lrow(Lk[k]) + c];
        }
    for (int j = w; j < M * PR; j += TW) {
        const int m = j % M;
        const float4* __restrict__ row = reinterpret_cast<const float4*>(a.ainv + (size_t)(blockIdx.x * M + m) * a.ndp);
        float s = 0.f;
#pragma unroll 4
        for (int k = (j / M) * 32 + lane; k < n4; k += 32 * PR) {
            const float4 v = __ldg(row + k), u = rc4[k];
            s += v.x * u.x + v.y * u.y + v.z * u.z + v.w * u.w;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) zs[j / M][m] = s;
    }
    __syncthreads();
    float zc[M], rz = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        zc[m] = 0.f;
#pragma unroll
        for (int k = 0; k < PR; ++k) zc[m] += zs[k][m];
        rz += zc[m] * a.rc[(size_t)blockIdx.x * M + m];
    }
    auto add_coarse = [&](const float4& L, const float (&zv)[NC]) {
        const size_t d = (size_t)NC * lrow(L);
        float o[NC];
        prolong<NC, M>(zc, L, o);
        const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (!((mk >> c) & 1)) a.z[d + c] = zv[c] + o[c];
    };
#pragma unroll
    for (int k = 0; k < CZ_KEEP; ++k)
        if (t0 + TW * 32 * k < t1) add_coarse(Lk[k], zk[k]);
    for (int t = t0 + TW * 32 * CZ_KEEP; t < t1; t += TW * 32) {
        const float4 L = __ldg(a.lnode + t);
        float zv[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) zv[c] = a.z[(size_t)NC * lrow(L) + c];
        add_coarse(L, zv);
    }
    if (threadIdx.x == 0) reinterpret_cast<float2*>(a.part)[blockIdx.x] = make_float2(rz, 0.f);
    if (!last_block(&S->ticket2)) return;
    const df tot = reduce_parts_df_sum(reinterpret_cast<const float2*>(a.part), gridDim.x);
    if (threadIdx.x != 0) return;
    S->ticket2 = 0;
    const df rz_new = df_add_acc(df{S->rzloc.x, S->rzloc.y}, tot), rz_old = {S->rz_old.x, S->rz_old.y};
    const double rzn = df_value(rz_new);
    S->absNew = rzn;
    S->rz_new = make_float2(rz_new.hi, rz_new.lo);
    if (MODE == CZ_UPDATE) S->beta = df_quotient(rz_new, rz_old);  // (through FP64 the tail takes 0.6 us more)
    else if (MODE == CZ_INIT) { S->absOld = rzn; S->rz_old = S->rz_new; S->beta = 0.0; }
    else {
        S->beta = S->fresh ? 0.0 : rzn / S->absOld;
        S->done = 0;
        S->rst = 0;
    }
    // not positive: the matrix or the inverse is not definite; the host solves one-level
    if (!(rz_new.hi > 0.f)) { S->bad = 1; S->done = 1; }
}

// q = A p and p.q for scalar rows: sliced ELL in aggregate order.
// The CTAs take contiguous runs of slices with the same number of slots (bnd),
// and the warps of a CTA contiguous runs of its slots, whatever slices these
// belong to: a warp that starts inside a slice leaves its sum to be added to
// the slice's (in warp order).  With one warp per slice the 16,608 slices of a
// P2 mesh took three rounds of 7,296 warps where 2.3 were work; all gathers of
// a batch come before its sums, as nothing moves across the tests for a
// slice's end.  531k rows of P2 tetrahedra: 42.5 -> 32-33 us with 8 or 12 slots
// in flight and 4 CTAs per SM; 41 us with 8 and 6, whose registers spill.
constexpr int SPMV_PER_SM = 4;
template <int U, typename TC>
__global__ void __launch_bounds__(256, SPMV_PER_SM) k_cz_spmv(CzSpmv m, const TC* __restrict__ col) {
    constexpr int NWP = 8, CAP = 32;
    CGScal* S = m.S;
    chain_next();
    chain_wait();
    if (S->done) return;
    __shared__ double sh[32];
    __shared__ int so[CAP + 1], hs[NWP];
    __shared__ float acc[CAP][32], head[NWP][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const float* p = m.p;
    float loc = 0.f;
    const int s1 = m.bnd[blockIdx.x + 1];
    for (int g0 = m.bnd[blockIdx.x]; g0 < s1; g0 += CAP) {
        const int gn = min(CAP, s1 - g0);
        if ((int)threadIdx.x <= gn) so[threadIdx.x] = m.soff[g0 + threadIdx.x] >> 5;
        for (int k = threadIdx.x; k < gn * 32; k += 256) (&acc[0][0])[k] = 0.f;
        if (lane == 0) hs[w] = -1;
        __syncthreads();
        const int T0 = so[0], T = so[gn] - T0;
        int k = T0 + (int)((long long)T * w / NWP);
        const int kend = T0 + (int)((long long)T * (w + 1) / NWP);
        if (k < kend) {
            int ls = 0;
            while (so[ls + 1] <= k) ++ls;
            bool inside = k > so[ls];
            int next = so[ls + 1];
            float a = 0.f;
            auto flush = [&] {
                if (inside && lane == 0) hs[w] = ls;
                (inside ? head[w] : acc[ls])[lane] = a;
                a = 0.f;
                inside = false;
            };
            for (; k < kend; k += U) {
                int j[U], li = ls, ln = next;
                float v[U], x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (k + u < kend) {
                        j[u] = ld_stream(col + (size_t)(k + u) * 32 + lane);
                        if (sizeof(TC) == 2) {
                            while (k + u >= ln) ln = so[++li + 1];
                            const int i = (g0 + li) * 32 + lane;
                            j[u] += i < m.nrow ? i : 0;
                        }
                        v[u] = ld_stream(m.val + (size_t)(k + u) * 32 + lane);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k + u < kend) x[u] = p[j[u]];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (k + u < kend) {
                        while (k + u >= next) {
                            flush();
                            next = so[++ls + 1];
                        }
                        a += v[u] * x[u];
                    }
                }
            }
            flush();
        }
        __syncthreads();
        for (int l = w; l < gn; l += NWP) {
            const int i = (g0 + l) * 32 + lane;
            if (i >= m.nrow) continue;
            float t = acc[l][lane];
#pragma unroll
            for (int h = 0; h < NWP; ++h)
                if (hs[h] == l) t += head[h][lane];
            m.q[i] = t;
            loc += p[i] * t;
        }
        __syncthreads();
    }
    const df bsum = block_sum_df(loc, reinterpret_cast<float*>(sh));
    if (threadIdx.x == 0) reinterpret_cast<float2*>(m.part)[blockIdx.x] = make_float2(bsum.hi, bsum.lo);
    if (last_block(&S->ticket1)) {
        const double tot = reduce_parts_df_blk<256>(reinterpret_cast<const float2*>(m.part), gridDim.x, sh);
        if (threadIdx.x == 0) {
            S->pAp = tot;
            S->alpha = S->absNew / tot;
            S->ticket1 = 0;
        }
    }
}

// first slice of every CTA of k_cz_spmv
__global__ void k_cz_bnd(int ncta, int nslice, const int* __restrict__ soff, int* __restrict__ bnd) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > ncta) return;
    const int64_t goal = (int64_t)soff[nslice] * b / ncta;
    int lo = 0, hi = nslice;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (soff[mid] < goal) lo = mid + 1;
        else hi = mid;
    }
    bnd[b] = lo;
}

// p = z + beta p (where the product does not fold the direction update)
__global__ void __launch_bounds__(256) k_cz_dir(int n, const float* z, float* p, const CGScal* S) {
    chain_next();
    chain_wait();
    if (S->done) return;
    const float beta = (float)S->beta;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) p[i] = fmaf(beta, p[i], z[i]);
}

// ---------------------------------------------------------------------------
// Small systems: the whole two-level solve in one thread-block cluster.  Every
// CTA owns whole aggregates (list order), with their vectors, inverse blocks
// and row lists in shared memory, and, with MS, its rows of the matrix too.
// An iteration has three cluster barriers: after the update (r.r, r.z, P^T r),
// after the coarse correction (its term of r.z; w = z + P z_c visible), and
// after the product with the folded direction p = w + beta p (p.q).  The sums
// travel as double-float pairs through distributed shared memory, each CTA
// storing its pair into every peer before the barrier, so that no CTA reads
// remotely after it.  The FP64 reliable updates run in the same launch.
// One iteration takes about a third of the three launches of the graph path,
// whose latency does not shrink with the system, and uses at most 16 SMs, so that
// concurrent solves run side by side.
namespace cgrp = cooperative_groups;

struct CzClu {
    const float4* lnode;
    const int *sofs, *cta, *perm;
    const float *dsub, *ainv;
    const CzInst* inst;
    const int* order;        // batch: the instance of every cluster
    int cta_stride;          // ... and the entries of cta per instance
    int inst_id;             // the instance, where order is null
    OlScal* res;             // batch: results (null: S)
    const int *rp, *ci;      // (block) CSR in list order
    const float* val;        // [NC * NC][nent]
    int nent;
    const float* dinv;       // node blocks: by natural row; scalar: in list order
    float *rc, *w, *pa, *pb; // P^T r (two buffers of ndp), w and the direction buffers, list order
    const int* aeq;          // equation of every component of a natural row (null: NC row + c)
    const double* b;
    double* x64;
    const int *rowptr, *colind;  // FP64 CSR by equation
    const double* val64;
    CGScal* S;
    double tol, drop;
    int max_iter, max_gap, exact64;
    float4* part;            // grid form: the CTAs' sums, four slots
    unsigned* bar;
    int inv_smem;            // the CTA's rows of the inverse are held in shared memory
    unsigned bar_start;      // grid form: count at which the barrier starts
};


template <int NC, int M, int NW>
size_t clu_smem(int rows, int aggs, int ndp, int ent, bool ms, bool as) {
    size_t f = (size_t)rows * (5 * NC + NC * NC + 4 + 1) + (size_t)aggs * (NW * M + M) + ndp + 8;
    f += (size_t)aggs * NW * M * M;             // sub-aggregate blocks
    if (as) f += (size_t)aggs * M * ndp;        // rows of the inverse
    if (ms) f += (size_t)ent * (NC * NC + 1) + rows + 1;
    return 4 * f + 64;
}

template <int NC, int M, int NW, int LPR, bool MS, bool GRID, int CLT>
__global__ void __launch_bounds__(CLT, 1) k_cz_cluster(CzClu a) {
    cgrp::cluster_group cl = cgrp::this_cluster();
    extern __shared__ __align__(16) float smem[];
    __shared__ float4 red[4][16];
    __shared__ float bs[2][32];
    __shared__ double shd[32];
    __shared__ float sc_alpha, sc_beta;
    __shared__ int sc_ctl;
    const int rank = GRID ? (int)blockIdx.x : (int)cl.block_rank(), ncta = GRID ? (int)gridDim.x : (int)cl.num_blocks();
    const int inst = !GRID && a.order ? a.order[blockIdx.x / ncta] : a.inst_id;
    const CzInst in = a.inst[inst];
    const int ndp = in.ndp;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int* cta = a.cta + (!GRID && a.order ? (size_t)inst * a.cta_stride : 0);
    const int ag0 = cta[rank], ag1 = cta[rank + 1], na = ag1 - ag0;
    const int c0 = (ag0 - in.agg0) * M;                // first coarse unknown of this CTA
    const float* ainv = a.ainv + in.a0 + (size_t)c0 * ndp;
    const int t0 = a.sofs[ag0 * NW], nr = a.sofs[ag1 * NW] - t0;
    const int R = in.rows, E = in.ent;
    float4* ln = reinterpret_cast<float4*>(smem);     // positions; w: aggregate (local), mask above
    float* rcs = smem + 4 * (size_t)R;                // [ndp], 16-byte aligned as ln
    float* ais = rcs + ndp;                           // [agg M][ndp]
    float* xs = ais + (a.inv_smem ? (size_t)in.aggs * M * ndp : 0);
    float* rs = xs + (size_t)NC * R;
    float* qs = rs + (size_t)NC * R;
    float* zs = qs + (size_t)NC * R;
    float* ps = zs + (size_t)NC * R;
    float* ds = ps + (size_t)NC * R;                  // [NC * NC][row]
    float* src = ds + (size_t)(NC * NC) * R;          // [sub][M]
    float* zcs = src + (size_t)in.aggs * NW * M;      // [agg][M]
    float* dss = zcs + (size_t)in.aggs * M;           // [sub][M * M]
    int* nat = reinterpret_cast<int*>(dss + (size_t)in.aggs * NW * M * M);  // natural row
    int* rps = nat + R;                               // MS: rows, columns, values
    int* cis = rps + R + 1;
    float* vs = reinterpret_cast<float*>(cis + E);
    for (int u = w; u < na * NW; u += CLT / 32) {
        const int s0 = a.sofs[ag0 * NW + u], s1 = a.sofs[ag0 * NW + u + 1];
        for (int t = s0 + lane; t < s1; t += 32) {
            float4 L = a.lnode[t];
            L.w = __int_as_float((u / NW) | (NC == 3 ? lmask(L) << ROW_BITS : 0));
            ln[t - t0] = L;
        }
    }
    for (int k = tid; a.inv_smem && k < na * M * (ndp / 4); k += CLT)
        reinterpret_cast<float4*>(ais)[k] = reinterpret_cast<const float4*>(ainv)[k];
    for (int k = tid; k < na * NW * M * M; k += CLT) dss[k] = a.dsub[(size_t)(ag0 * NW) * (M * M) + k];
    const int e0 = a.rp[t0];
    for (int i = tid; i < nr; i += CLT) {
        const int row = a.perm[t0 + i];
        nat[i] = row;
#pragma unroll
        for (int k = 0; k < NC * NC; ++k) ds[k * R + i] = NC == 1 ? a.dinv[t0 + i] : a.dinv[(size_t)9 * row + k];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            xs[NC * i + c] = 0.f;
            ps[NC * i + c] = 0.f;
            qs[NC * i + c] = 0.f;
            a.pa[(size_t)NC * (t0 + i) + c] = 0.f;
        }
    }
    if (MS) {
        const int ne = a.rp[t0 + nr] - e0;
        for (int i = tid; i <= nr; i += CLT) rps[i] = a.rp[t0 + i] - e0;
        for (int k = tid; k < ne; k += CLT) {
            cis[k] = a.ci[e0 + k];
#pragma unroll
            for (int e = 0; e < NC * NC; ++e) vs[(size_t)e * E + k] = a.val[(size_t)e * a.nent + e0 + k];
        }
    }
    int slot = 0;
    bool alive = true;  // grid form: false in every thread once a barrier has timed out
    GridBarrier gb(a.bar, &a.S->fault, a.bar_start);
    auto sync_all = [&]() {
        if constexpr (GRID) alive = gb.sync();
        else cl.sync();
    };
    // sums over all CTAs of u, and of v if TWO: valid in thread 0 of every CTA.
    // FP32 inside a warp, double-float from there.
    auto cl_sum = [&](auto two, float u, float v, df& ou, df& ov) {
        constexpr bool TWO = decltype(two)::value;
        for (int o = 16; o > 0; o >>= 1) {
            u += __shfl_xor_sync(0xffffffffu, u, o);
            if (TWO) v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (lane == 0) { bs[0][w] = u; if (TWO) bs[1][w] = v; }
        __syncthreads();
        if (w == 0) {
            ou = {lane < CLT / 32 ? bs[0][lane] : 0.f, 0.f};
            ov = {TWO && lane < CLT / 32 ? bs[1][lane] : 0.f, 0.f};
            warp_sum_df2<TWO, true, CLT / 64>(ou, ov);
            const float4 t = make_float4(ou.hi, ou.lo, ov.hi, ov.lo);
            if constexpr (GRID) {
                if (lane == 0) __stcg(a.part + slot * ncta + rank, t);
            } else {
                if (lane < ncta) *cl.map_shared_rank(&red[slot][rank], lane) = t;
            }
        }
        sync_all();
        if (w == 0) {
            ou = ov = {0.f, 0.f};
            if constexpr (GRID) {
                for (int base = 0; base < ncta; base += 160) {
                    float4 r[5];
#pragma unroll
                    for (int k = 0; k < 5; ++k) {
                        const int i = base + 32 * k + lane;
                        r[k] = i < ncta ? __ldcg(a.part + slot * ncta + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int k = 0; k < 5; ++k) {
                        ou = df_add_acc(ou, df{r[k].x, r[k].y});
                        if (TWO) ov = df_add_acc(ov, df{r[k].z, r[k].w});
                    }
                }
            } else if (lane < ncta) {
                const float4 r = red[slot][lane];
                ou = {r.x, r.y};
                ov = {r.z, r.w};
            }
            warp_sum_df2<TWO, false, GRID ? 16 : 8>(ou, ov);  // (a cluster has 16 CTAs at most)
        }
        slot = (slot + 1) & 3;
    };
    auto cl_sum_d = [&](double u, double& o) {  // one FP64 value (rare)
        const double t = block_sum(u, shd);
        if (w == 0) {
            const double tt = __shfl_sync(0xffffffffu, t, 0);
            if constexpr (GRID) {
                if (lane == 0) __stcg(reinterpret_cast<double*>(a.part + slot * ncta + rank), tt);
            } else {
                if (lane < ncta) *reinterpret_cast<double*>(cl.map_shared_rank(&red[slot][rank], lane)) = tt;
            }
        }
        sync_all();
        o = 0.0;
        if (w == 0) {
            double r = 0.0;
            if constexpr (GRID) {
                for (int i = lane; i < ncta; i += 32) r += __ldcg(reinterpret_cast<const double*>(a.part + slot * ncta + i));
            } else if (lane < ncta) {
                r = *reinterpret_cast<const double*>(&red[slot][lane]);
            }
            for (int k = 16; k > 0; k >>= 1) r += __shfl_xor_sync(0xffffffffu, r, k);
            o = r;
        }
        slot = (slot + 1) & 3;
    };
    // scalars, held by thread 0 of every CTA (the same values everywhere)
    df rz = {0.f, 0.f}, rz_old = {0.f, 0.f}, rzl = {0.f, 0.f};
    double rr = 0.0, thr = 0.0, trig = 0.0, rr_true = 0.0, rr_last = 0.0, rr_best = 0.0, bn = 0.0;
    int iters = 0, last_upd = 0, stall = 0, careful = 0;
    enum { GO = 0, FIN1 = 1, FIN2 = 2, FIN3 = 3, STOP = 4 };

    // z = D0^-1 r + P_s D_s^-1 P_s^T r from rs, with rr and rz of this thread; rc written
    int par = 0;
    // (a restart's r.z in FP64, in drz)
    auto local_part = [&](float alpha, bool update, float& frr, float& frz, double& drz) {
        for (int u = w; u < na * NW; u += CLT / 32) {
            const int sub = ag0 * NW + u;
            const int i0 = a.sofs[sub] - t0, i1 = a.sofs[sub + 1] - t0;
            float rc[M];
#pragma unroll
            for (int m = 0; m < M; ++m) rc[m] = 0.f;
            for (int i = i0 + lane; i < i1; i += 32) {
                float rv[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    rv[c] = rs[NC * i + c];
                    if (update) {
                        xs[NC * i + c] += alpha * ps[NC * i + c];
                        rv[c] -= alpha * qs[NC * i + c];
                        rs[NC * i + c] = rv[c];
                    }
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    float z = 0.f;
#pragma unroll
                    for (int k = 0; k < NC; ++k) z += ds[(NC * c + k) * R + i] * rv[k];
                    zs[NC * i + c] = z;
                    if (update) {
                        frr += rv[c] * rv[c];
                        frz += rv[c] * z;
                    } else {
                        drz += (double)rv[c] * (double)z;
                    }
                }
                restrict_add<NC, M>(rc, rv, ln[i]);
            }
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) rc[m] += __shfl_xor_sync(0xffffffffu, rc[m], o);
            float z1[M], rz1 = 0.f;
            const float* D = dss + (size_t)u * (M * M);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                z1[m] = 0.f;
#pragma unroll
                for (int k = 0; k < M; ++k) z1[m] += D[M * m + k] * rc[k];
                rz1 += rc[m] * z1[m];
            }
            if (lane == 0) {
                if (update) frz += rz1;
                else drz += (double)rz1;
#pragma unroll
                for (int m = 0; m < M; ++m) src[u * M + m] = rc[m];
            }
            for (int i = i0 + lane; i < i1; i += 32) {
                float o[NC];
                const float4 L = ln[i];
                prolong<NC, M>(z1, L, o);
                const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    if (!((mk >> c) & 1)) zs[NC * i + c] += o[c];
            }
        }
        __syncthreads();
        float* rcg = a.rc + in.rc0 + (size_t)par * ndp;
        for (int k = tid; k < na * M; k += CLT) {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < NW; ++j) s += src[((k / M) * NW + j) * M + k % M];
            rcg[c0 + k] = s;
        }
    };
    // after the barrier that made P^T r visible: w = z + P A_c^-1 P^T r (own rows);
    // this CTA's part of the coarse term of r.z in thread 0's return value
    auto coarse_part = [&]() -> float {
        const float* rcg = a.rc + in.rc0 + (size_t)par * ndp;
        for (int k = tid; k < ndp; k += CLT) rcs[k] = rcg[k];
        par ^= 1;
        __syncthreads();
        const int n4 = ndp / 4;
        const float4* rc4 = reinterpret_cast<const float4*>(rcs);
        float part = 0.f;
        for (int k = w; k < na * M; k += CLT / 32) {
            const float4* row = reinterpret_cast<const float4*>((a.inv_smem ? ais : ainv) + (size_t)k * ndp);
            float s = 0.f;
#pragma unroll 4
            for (int j = lane; j < n4; j += 32) {
                const float4 v = row[j], u = rc4[j];
                s += v.x * u.x + v.y * u.y + v.z * u.z + v.w * u.w;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) {
                zcs[k] = s;
                part += s * rcs[c0 + k];
            }
        }
        __syncthreads();
        for (int i = tid; i < nr; i += CLT) {
            const float4 L = ln[i];
            float c6[M], o[NC];
            const int ag = lrow(L);
#pragma unroll
            for (int m = 0; m < M; ++m) c6[m] = zcs[ag * M + m];
            prolong<NC, M>(c6, L, o);
            const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float z = zs[NC * i + c] + ((mk >> c) & 1 ? 0.f : o[c]);
                a.w[(size_t)NC * (t0 + i) + c] = z;
                zs[NC * i + c] = z;
            }
        }
        return part;
    };

    sync_all();  // every CTA runs: its shared memory may be written
    if (!alive) return;
    // start: r = b
    {
        double bb = 0.0;
        for (int i = tid; i < nr; i += CLT)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int e = a.aeq ? a.aeq[NC * nat[i] + c] : NC * nat[i] + c;
                const double v = e >= 0 ? a.b[e] : 0.0;
                rs[NC * i + c] = (float)v;
                bb += v * v;
                if (e >= 0) a.x64[e] = 0.0;
            }
        __syncthreads();
        double t;
        cl_sum_d(bb, t);
        if (!alive) return;
        if (tid == 0) {
            bn = rr_true = rr_best = rr = t;
            thr = a.tol * a.tol * t;
            trig = a.drop * t;
            sc_ctl = !(t == t) ? FIN3 : (t == 0.0 ? FIN1 : GO);
        }
        __syncthreads();
    }
    int ctl = sc_ctl;
    bool restart = true, fresh = true;  // the first pass starts like a restart with beta = 0
    const int lr = tid % LPR, grp = tid / LPR;
    constexpr int NG = CLT / LPR;
    float alpha = 0.f;
    while (ctl == GO) {
        df s0 = {0.f, 0.f}, s1 = {0.f, 0.f};
        float frr = 0.f, frz = 0.f;
        double drz = 0.0;
        local_part(alpha, !restart, frr, frz, drz);
        if (restart) {
            cl_sum_d(drz, drz);
            s1 = df_from_double(drz);
        } else {
            cl_sum(std::true_type{}, frr, frz, s0, s1);
        }
        if (!alive) return;
        if (tid == 0) {
            int k = GO;
            rzl = s1;
            if (!restart) {
                rr = df_value(s0);
                iters += 1;
                rz_old = rz;
                if (!(rr == rr) || !(s1.hi == s1.hi)) k = FIN3;
                else if (rr < thr || rr < trig || (a.exact64 && rr > 1e8 * rr_true) || iters >= a.max_iter) k = STOP;
                else if (a.exact64 && iters - last_upd >= a.max_gap) k = FIN3;
            }
            sc_ctl = k;
        }
        __syncthreads();
        ctl = sc_ctl;
        if (ctl == FIN3) break;
        if (ctl == STOP) {
            // fold the increment, then the FP64 residual
            for (int i = tid; i < nr; i += CLT)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const int e = a.aeq ? a.aeq[NC * nat[i] + c] : NC * nat[i] + c;
                    if (e >= 0) a.x64[e] += (double)xs[NC * i + c];
                    xs[NC * i + c] = 0.f;
                }
            if (!a.exact64) {
                __syncthreads();  // every thread has read the code that thread 0 replaces
                if (tid == 0) { sc_ctl = rr < thr ? FIN1 : FIN2; rr_true = rr; }
                __syncthreads();
                ctl = sc_ctl;
                break;
            }
            sync_all();
            if (!alive) return;
            double loc = 0.0;
            for (int base = grp - grp % (32 / LPR); base < nr * NC; base += NG) {  // warp-uniform
                const int k = base + grp % (32 / LPR);
                const bool act = k < nr * NC;
                int e = -1;
                if (act) e = a.aeq ? a.aeq[NC * nat[k / NC] + k % NC] : NC * nat[k / NC] + k % NC;
                double acc = 0.0;
                if (e >= 0)
                    for (int j = a.rowptr[e] + lr; j < a.rowptr[e + 1]; j += LPR) acc += __ldg(a.val64 + j) * a.x64[__ldg(a.colind + j)];
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, LPR);
                if (act && lr == 0) {
                    const double ri = e >= 0 ? a.b[e] - acc : 0.0;
                    rs[k] = (float)ri;
                    loc += ri * ri;
                }
            }
            double t;
            cl_sum_d(loc, t);
            if (!alive) return;
            if (tid == 0) {
                int k = GO;
                last_upd = iters;
                if (!(t == t)) k = FIN3;
                else {
                    const double rec = rr;
                    rr_true = t;
                    if (t <= thr) k = FIN1;
                    else if (iters >= a.max_iter) k = FIN2;
                    else {
                        stall = t > 0.81 * rr_best ? stall + 1 : 0;
                        rr_best = fmin(rr_best, t);
                        if (stall >= 6) k = FIN3;
                        fresh = rr_last > 0.0 && t >= rr_last;
                        rr_last = t;
                        if (t > 2.0 * rec) careful = 1;
                        trig = (!careful && t < 1.003 * rec ? a.drop * a.drop : a.drop) * t;
                    }
                }
                sc_ctl = k;
            }
            __syncthreads();
            ctl = sc_ctl;
            restart = true;
            continue;
        }
        const float cp = coarse_part();
        cl_sum(std::false_type{}, cp, 0.f, s0, s1);
        if (!alive) return;
        if (tid == 0) {
            rz = df_add_acc(rzl, s0);
            const bool first = rz_old.hi == 0.f;
            sc_beta = (restart && (fresh || first)) ? 0.f : df_quotient(rz, rz_old);
            sc_ctl = rz.hi > 0.f ? GO : FIN3;  // also when it is not a number
            fresh = false;
        }
        __syncthreads();
        ctl = sc_ctl;
        if (ctl != GO) break;
        restart = false;
        // p = w + beta p, q = A p
        const float beta = sc_beta;
        const float* pold = a.pa;
        float* pnew = a.pb;
        float loc = 0.f;
        for (int base = grp - grp % (32 / LPR); base < nr; base += NG) {
            const int i = base + grp % (32 / LPR);
            const bool act = i < nr;
            float acc[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[c] = 0.f;
            int k = 0, k1 = 0;
            if (act) {
                k = (MS ? rps[i] : a.rp[t0 + i]) + lr;
                k1 = MS ? rps[i + 1] : a.rp[t0 + i + 1];
            }
#pragma unroll 2
            for (; k < k1; k += LPR) {
                const size_t j = (size_t)NC * (MS ? cis[k] : __ldg(a.ci + k));
                float x[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) x[c] = fmaf(beta, pold[j + c], a.w[j + c]);
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int e = 0; e < NC; ++e)
                        acc[c] += (MS ? vs[(size_t)(NC * c + e) * E + k] : __ldg(a.val + (size_t)(NC * c + e) * a.nent + k)) * x[e];
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o, LPR);
            if (act && lr == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float p = fmaf(beta, ps[NC * i + c], zs[NC * i + c]);  // the bits the gathers form
                    ps[NC * i + c] = p;
                    pnew[(size_t)NC * (t0 + i) + c] = p;
                    qs[NC * i + c] = acc[c];
                    loc += p * acc[c];
                }
            }
        }
        { float* sw = a.pa; a.pa = a.pb; a.pb = sw; }  // the buffer just written is read next time
        cl_sum(std::false_type{}, loc, 0.f, s0, s1);
        if (!alive) return;
        if (tid == 0) sc_alpha = df_quotient(rz, s0);
        __syncthreads();
        alpha = sc_alpha;
    }
    if (rank == 0 && tid == 0 && a.res) {
        OlScal* S = a.res + inst;
        S->fin = ctl;
        S->iters = iters;
        S->rr = rr_true;
        S->rhs2 = bn;
    } else if (rank == 0 && tid == 0) {
        CGScal* S = a.S;
        S->fin = ctl;
        S->iters = iters;
        S->rr_true = rr_true;
        S->rhsNorm2 = bn;
        S->rr = rr;
    }
    if constexpr (!GRID) cl.sync();  // no CTA leaves while a peer can still store into it
}

// ---------------------------------------------------------------------------
// Numeric setup, once per assembly

// instance of a row
__device__ inline int inst_of(const CzInst* __restrict__ inst, int ninst, int row) {
    int lo = 0, hi = ninst;  // the last one that starts at or before the row (empty ones start where the next does)
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (inst[mid].row0 <= row) lo = mid;
        else hi = mid;
    }
    return lo;
}

// largest diagonal entry of every aggregate, and (top) of every instance (positive floats order as integers)
template <int NC, int NW, typename T>
__global__ void __launch_bounds__(NW * 32) k_cz_amax(const int* __restrict__ sofs, const int* __restrict__ perm,
                                                     const int* __restrict__ aeq, const int* __restrict__ diag,
                                                     const T* __restrict__ val, const int* __restrict__ agg_inst,
                                                     float* __restrict__ out, float* __restrict__ top) {
    __shared__ float sh[NW];
    float m = 0.f;
    for (int t = sofs[blockIdx.x * NW] + blockIdx.y * NW * 32 + threadIdx.x; t < sofs[(blockIdx.x + 1) * NW]; t += gridDim.y * NW * 32) {
        const int row = perm[t];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int e = NC == 3 && aeq ? aeq[NC * row + c] : NC * row + c;
            const float v = e >= 0 ? fabsf((float)val[diag[e]]) : 0.f;
            if (v < INFINITY) m = fmaxf(m, v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < NW; ++w) m = fmaxf(m, sh[w]);
    atomicMax(reinterpret_cast<int*>(out + blockIdx.x), __float_as_int(m));
    atomicMax(reinterpret_cast<int*>(top + agg_inst[blockIdx.x]), __float_as_int(m));
}

// Fixed point of the coarse entries between two aggregates, from their largest
// diagonal entries: |a_ij| <= sqrt(a_ii a_jj) < 2^e, and 2^FIX_BITS stands for
// 2^e.  (One scale for the whole matrix loses the couplings of a soft region to
// rounding: with a contrast of 1e8 its coarse matrix was noise, and the solve
// fell back to one-level after 160^2 Q1 iterations that now end after 52.)
// 0: the couplings of an aggregate softer than 2^-30 of the stiffest (top) are
// left out, which keeps the matrix definite.  With them the FP32 directions
// hold amplitudes of both regions, and lose the stiff one's: 20^3 P2
// tetrahedra with one half softer by 1e8 take 160 iterations (402 one-level), by
// 1e9 291, by 1e10 1,057, without them 173 and 175; 160^2 Q1 takes 52 whatever the
// contrast, without them 165.
constexpr float SOFT = 1.f / (1 << 30);
__device__ inline float fix_scale(float amax_i, float amax_j, float top) {
    if (fminf(amax_i, amax_j) < SOFT * top) return 0.f;
    const int e = ((__float_as_int(amax_i) >> 23) + (__float_as_int(amax_j) >> 23) - 2 * 126 + 1) >> 1;
    return __int_as_float((min(126, FIX_BITS - e) + 127) << 23);
}

// Galerkin blocks: CTA per aggregate, warp per sub-aggregate, lane per row.
// The entries inside a sub-aggregate and inside the aggregate are summed in
// registers and by fixed shuffle trees; those towards a later aggregate go to
// acc in fixed point, one run of equal aggregates of a row at a time (the
// entries towards earlier ones follow by symmetry).
template <int NC, int M, int NW>
__global__ void __launch_bounds__(NW * 32) k_cz_galerkin(CzMat A, const float4* __restrict__ lnode, const float4* __restrict__ yrow,
                                                         const int* __restrict__ sofs, const CzInst* __restrict__ inst,
                                                         const int* __restrict__ agg_inst, const float* __restrict__ amax,
                                                         const float* __restrict__ top,
                                                         unsigned long long* __restrict__ acc, float* __restrict__ dsub,
                                                         float* __restrict__ dagg) {
    __shared__ float own[NW][M * M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x, sub = I * NW + w;
    const int ik = agg_inst[I], ndp = inst[ik].ndp, agg0 = inst[ik].agg0;
    acc += inst[ik].a0;
    float a1[M * M], a2[M * M];
#pragma unroll
    for (int k = 0; k < M * M; ++k) a1[k] = a2[k] = 0.f;
    // B_i^T T for the row's modes B_i and T [NC][M]
    auto outer = [](const float (&T)[NC][M], const float4& y, float (&o)[M * M], bool add) {
#pragma unroll
        for (int b = 0; b < M; ++b) {
            float col[NC], rc[M];
#pragma unroll
            for (int c = 0; c < NC; ++c) col[c] = T[c][b];
#pragma unroll
            for (int m = 0; m < M; ++m) rc[m] = 0.f;
            restrict_add<NC, M>(rc, col, y);
#pragma unroll
            for (int m = 0; m < M; ++m) o[m * M + b] = add ? o[m * M + b] + rc[m] : rc[m];
        }
    };
    for (int t = sofs[sub] + lane; t < sofs[sub + 1]; t += 32) {
        const float4 L = lnode[t];
        const int i = lrow(L);
        float T1[NC][M], T2[NC][M], Tc[NC][M];
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int m = 0; m < M; ++m) T1[c][m] = T2[c][m] = Tc[c][m] = 0.f;
        int J = I;  // aggregate of the run in Tc (I: none)
        auto flush = [&]() {
            float o[M * M];
            const float scale = fix_scale(amax[I], amax[J], top[ik]);
            outer(Tc, L, o, false);
            unsigned long long* dst = acc + (size_t)((I - agg0) * M) * ndp + (size_t)(J - agg0) * M;
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int b = 0; b < M; ++b)
                    atomicAdd(dst + (size_t)m * ndp + b, (unsigned long long)__float2ll_rn(o[m * M + b] * scale));
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int m = 0; m < M; ++m) Tc[c][m] = 0.f;
        };
        int k0, k1, step;
        if (NC == 3 || A.soff) {
            const int s = i >> 5;
            k0 = A.soff[s] + (i & 31);
            k1 = k0 + 32 * A.swid[s];
            step = 32;
        } else {
            k0 = A.rowptr[i];
            k1 = A.rowptr[i + 1];
            step = 1;
        }
        for (int k = k0; k < k1; k += step) {
            const int j = A.col[k];
            const float4 y = __ldg(yrow + j);
            const int sj = __float_as_int(y.w), Jj = sj / NW;
            if (Jj < I) continue;
            float v[NC * NC];
            if (NC == 3) {
                const float* vp = A.val + (size_t)(k >> 5) * 288 + (k & 31);
#pragma unroll
                for (int e = 0; e < NC * NC; ++e) v[e] = vp[32 * e];
            } else {
                v[0] = A.val[k];
            }
            if (Jj != I && Jj != J) {
                if (J != I) flush();
                J = Jj;
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float row[NC], tm[M];
#pragma unroll
                for (int e = 0; e < NC; ++e) row[e] = v[NC * c + e];
#pragma unroll
                for (int m = 0; m < M; ++m) tm[m] = 0.f;
                restrict_add<NC, M>(tm, row, y);  // row c of A_ij B_j
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    T1[c][m] += sj == sub ? tm[m] : 0.f;
                    T2[c][m] += (Jj == I && sj != sub) ? tm[m] : 0.f;
                    Tc[c][m] += Jj != I ? tm[m] : 0.f;
                }
            }
        }
        if (J != I) flush();
        outer(T1, L, a1, true);
        outer(T2, L, a2, true);
    }
#pragma unroll
    for (int k = 0; k < M * M; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a1[k] += __shfl_xor_sync(0xffffffffu, a1[k], o);
            a2[k] += __shfl_xor_sync(0xffffffffu, a2[k], o);
        }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < M * M; ++k) {
            dsub[(size_t)sub * (M * M) + k] = a1[k];
            own[w][k] = a1[k] + a2[k];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < M * M; k += NW * 32) {
        float s = 0.f;
        for (int v = 0; v < NW; ++v) s += own[v][k];
        dagg[(size_t)I * (M * M) + k] = s;
    }
}

// D_s^-1 in place: symmetric scaling, a small diagonal shift, Gauss-Jordan;
// modes without a positive diagonal (empty sub-aggregates, modes that vanish
// on one node) are left out
template <int M>
__global__ void k_cz_sub_inv(int nsub, float* __restrict__ dsub) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nsub) return;
    float* g = dsub + (size_t)t * (M * M);
    float A[M][M], s[M], dmax = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) dmax = fmaxf(dmax, g[m * M + m]);
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const float d = g[m * M + m];
        s[m] = d > 1e-6f * dmax ? rsqrtf(d) : 0.f;
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int k = 0; k < M; ++k)
            A[m][k] = m == k ? 1.f + REG : 0.5f * (g[m * M + k] + g[k * M + m]) * s[m] * s[k];
#pragma unroll
    for (int p = 0; p < M; ++p) {
        const float ip = 1.f / fmaxf(A[p][p], REG);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            if (m == p) continue;
            const float f = A[m][p] * ip;
#pragma unroll
            for (int k = 0; k < M; ++k)
                if (k != p) A[m][k] -= f * A[p][k];
            A[m][p] = -f;
        }
#pragma unroll
        for (int k = 0; k < M; ++k)
            if (k != p) A[p][k] *= ip;
        A[p][p] = ip;
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int k = 0; k < M; ++k) g[m * M + k] = 0.5f * (A[m][k] + A[k][m]) * s[m] * s[k];
}

// scaling of the coarse matrix to a unit diagonal (0: mode left out)
template <int M>
__global__ void k_cz_scale(int nagg, const float* __restrict__ dagg, float* __restrict__ s) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nagg) return;
    float dmax = 0.f;
    for (int m = 0; m < M; ++m) dmax = fmaxf(dmax, dagg[(size_t)t * (M * M) + m * M + m]);
    for (int m = 0; m < M; ++m) {
        const float d = dagg[(size_t)t * (M * M) + m * M + m];
        s[t * M + m] = d > 1e-6f * dmax ? rsqrtf(d) : 0.f;
    }
}

// the scaled coarse matrix of every instance, padded with the identity to whole tiles
template <int M>
__global__ void k_cz_form(const CzInst* __restrict__ inst, const unsigned long long* __restrict__ acc, const float* __restrict__ dagg,
                          const float* __restrict__ s, const float* __restrict__ amax, const float* __restrict__ top,
                          float* __restrict__ A) {
    const CzInst in = inst[blockIdx.z];
    const int nd = in.nd, ndp = in.ndp;
    if ((int)blockIdx.x * 32 >= ndp || (int)blockIdx.y * 32 >= ndp) return;
    acc += in.a0;
    A += in.a0;
    dagg += (size_t)in.agg0 * (M * M);
    s += in.agg0 * M;
    amax += in.agg0;
    const int j = blockIdx.x * 32 + (threadIdx.x & 31);
    for (int i = blockIdx.y * 32 + (threadIdx.x >> 5); i < (int)blockIdx.y * 32 + 32; i += 8) {
        float v = 0.f;
        if (i == j) v = 1.f + REG;
        else if (i < nd && j < nd) {
            const int I = i / M, J = j / M;
            if (I == J) v = 0.5f * (dagg[(size_t)I * M * M + (i % M) * M + j % M] + dagg[(size_t)I * M * M + (j % M) * M + i % M]);
            else if (const float f = fix_scale(amax[I], amax[J], top[blockIdx.z]); f > 0.f)
                v = (float)(long long)acc[I < J ? (size_t)i * ndp + j : (size_t)j * ndp + i] / f;
            v *= s[i] * s[j];
        }
        A[(size_t)i * ndp + j] = v;
    }
}

// Dense inversion of the coarse matrix (symmetric positive definite, unit
// diagonal) by block sweeps without pivoting, TB rows per step.  Sweeping
// block k takes A_kk to -D^-1, A_Ik to G_I = A_Ik D^-1 and A_IJ to
// A_IJ - G_I A_Jk^T, keeps the matrix symmetric, and leaves -A^-1 after the
// last block; only the tiles on and below the diagonal are stored.
//
// One launch per step, one CTA per tile.  Every CTA reads the panel (the tiles
// A_Ik) from a copy that the step before wrote, forms its own G_I, and the
// CTAs of the next panel's tiles write the next copy.  The next diagonal tile
// is also inverted by the CTA that updates it, beside the other tiles'
// updates: that chain, TB pivots with one block barrier each, is what a step
// waits for.  Measured at 64^3 (1,764 rows, 28 steps): see numeric().

// inverse of the TB x TB matrix in X by 256 threads, Gauss-Jordan: thread
// (ty, tx) holds rows ty + 16 r and columns tx + 16 c; pivot 16 a + b belongs to
// r = c = a, so that the registers are indexed by unrolled loops only.  The mean
// with its transpose is returned: an inverse that is symmetric only up to
// rounding turned the sweeps of a matrix with a condition of 1e5 (a contrast of
// 1e6 inside the aggregates) indefinite, its smallest eigenvalue -20 where 0.24
// was exact; with the symmetric one it stays 0.24.
__device__ __forceinline__ void tile_inv(float (*X)[TB + 1], float (*buf)[2 * TB]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float d[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) d[r][c] = X[ty + 16 * r][tx + 16 * c];
#pragma unroll
    for (int a = 0; a < 4; ++a)
        for (int b = 0; b < 16; ++b) {
            float* row = buf[b & 1];
            float* col = row + TB;
            if (ty == b) {
#pragma unroll
                for (int c = 0; c < 4; ++c) row[tx + 16 * c] = d[a][c];
            }
            if (tx == b) {
#pragma unroll
                for (int r = 0; r < 4; ++r) col[ty + 16 * r] = d[r][a];
            }
            __syncthreads();
            const float ip = __fdividef(1.f, fmaxf(row[16 * a + b], 0.1f * REG));
            float pr[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) pr[c] = row[tx + 16 * c];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float f = col[ty + 16 * r] * ip;
                const bool prow = r == a && ty == b;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const bool pcol = c == a && tx == b;
                    const float v = pcol ? -f : d[r][c] - f * pr[c];
                    d[r][c] = prow ? (pcol ? ip : pr[c] * ip) : v;
                }
            }
        }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) X[ty + 16 * r][tx + 16 * c] = d[r][c];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) d[r][c] = 0.5f * (d[r][c] + X[tx + 16 * c][ty + 16 * r]);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) X[ty + 16 * r][tx + 16 * c] = d[r][c];
    __syncthreads();
}

// o[r][c] = sum_m X[4 ty + r][m] Y[tx + 16 c][m]
__device__ __forceinline__ void tile_mul(const float (*X)[TB + 1], const float (*Y)[TB + 1], float (&o)[4][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) o[r][c] = 0.f;
#pragma unroll 8
    for (int m = 0; m < TB; ++m) {
        float u[4], v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) { u[r] = X[4 * ty + r][m]; v[r] = Y[tx + 16 * r][m]; }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[r][c] += u[r] * v[c];
    }
}

// a TB x TB tile (row stride ld) into shared memory
__device__ __forceinline__ void tile_load(const float* g, int ld, float (*X)[TB + 1]) {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int e = threadIdx.x + 256 * k;
        v[k] = *reinterpret_cast<const float4*>(g + (size_t)(e / 16) * ld + 4 * (e % 16));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int e = threadIdx.x + 256 * k, r = e / 16, c = 4 * (e % 16);
        X[r][c] = v[k].x; X[r][c + 1] = v[k].y; X[r][c + 2] = v[k].z; X[r][c + 3] = v[k].w;
    }
}

// the first panel and the inverse of the first diagonal tile
__global__ void __launch_bounds__(256) k_gj_first(const CzInst* __restrict__ inst, const float* __restrict__ A, float* __restrict__ panel) {
    __shared__ float X[TB][TB + 1];
    __shared__ float buf[2][2 * TB];
    const CzInst in = inst[blockIdx.y];
    const int n = in.ndp, I = blockIdx.x;
    if (I * TB >= n) return;
    A += in.a0;
    float *P = panel + in.p0, *Dinv = P + (size_t)2 * TB * n;
    tile_load(A + (size_t)(I * TB) * n, n, X);
    __syncthreads();
    for (int e = threadIdx.x; e < TB * TB; e += 256) P[(size_t)I * TB * TB + e] = X[e / TB][e % TB];
    if (I) return;
    tile_inv(X, buf);
    for (int e = threadIdx.x; e < TB * TB; e += 256) Dinv[e] = X[e / TB][e % TB];
}

__global__ void __launch_bounds__(256) k_gj_step(const CzInst* __restrict__ inst, int k, float* __restrict__ A, float* __restrict__ panel) {
    extern __shared__ __align__(16) float gj_smem[];
    typedef float (*Tile)[TB + 1];
    Tile X = reinterpret_cast<Tile>(gj_smem), Y = X + TB, Z = Y + TB;
    __shared__ float buf[2][2 * TB];
    const CzInst in = inst[blockIdx.y];
    const int n = in.ndp, nt = n / TB;
    if (k >= nt || (int)blockIdx.x >= nt * (nt + 1) / 2) return;
    A += in.a0;
    panel += in.p0;
    const float* P = panel + (size_t)(k & 1) * TB * n;
    float* Pnext = panel + (size_t)((k + 1) & 1) * TB * n;
    const float* Dinv = panel + (size_t)2 * TB * n + (k & 1) * TB * TB;
    float* Dnext = panel + (size_t)2 * TB * n + ((k + 1) & 1) * TB * TB;
    // tile (I, J), J <= I, of the linear index; the next diagonal tile comes first
    int t = blockIdx.x;
    const int first = k + 1 < nt ? (k + 1) * (k + 2) / 2 + k + 1 : -1;
    if (first >= 0) t = t == 0 ? first : (t <= first ? t - 1 : t);
    int I = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    while (I * (I + 1) / 2 > t) --I;
    const int J = t - I * (I + 1) / 2, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float* g = A + (size_t)(I * TB) * n + J * TB;
    float v[4][4];  // the tile's new entries, rows 4 ty + r, columns tx + 16 c
    if (I == k && J == k) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) v[r][c] = -Dinv[(4 * ty + r) * TB + tx + 16 * c];
    } else {
        // I == k: the tile is G_J^T
        const int R = I == k ? J : I;
        tile_load(P + (size_t)R * TB * TB, TB, X);
        tile_load(Dinv, TB, Y);
        float a[4][4];
        if (I != k && J != k) {
            tile_load(P + (size_t)J * TB * TB, TB, Z);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) a[r][c] = g[(size_t)(4 * ty + r) * n + tx + 16 * c];
        }
        __syncthreads();
        float o[4][4];
        tile_mul(X, Y, o);  // G_R: D^-1 is symmetric
        __syncthreads();
        if (I == k) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) X[tx + 16 * c][4 * ty + r] = o[r][c];
            __syncthreads();
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) v[r][c] = X[4 * ty + r][tx + 16 * c];
        } else if (J == k) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) v[r][c] = o[r][c];
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) X[4 * ty + r][tx + 16 * c] = o[r][c];
            __syncthreads();
            tile_mul(X, Z, o);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) v[r][c] = a[r][c] - o[r][c];
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) g[(size_t)(4 * ty + r) * n + tx + 16 * c] = v[r][c];
    // the next panel, column k + 1: tiles (I, k + 1), and (k + 1, J) transposed
    if (J == k + 1) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) Pnext[(size_t)I * TB * TB + (4 * ty + r) * TB + tx + 16 * c] = v[r][c];
    } else if (I == k + 1) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) Pnext[(size_t)J * TB * TB + (tx + 16 * c) * TB + 4 * ty + r] = v[r][c];
    }
    if (I != J || I != k + 1) return;
    __syncthreads();  // the next diagonal tile: its inverse
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) X[4 * ty + r][tx + 16 * c] = v[r][c];
    __syncthreads();
    tile_inv(X, buf);
    for (int e = threadIdx.x; e < TB * TB; e += 256) Dnext[e] = X[e / TB][e % TB];
}
constexpr int GJ_SMEM = 3 * TB * (TB + 1) * 4;

// undo the sign and the scaling, and fill the upper triangle from the lower
template <int M>
__global__ void k_cz_unscale(const CzInst* __restrict__ inst, const float* __restrict__ A, const float* __restrict__ s,
                             float* __restrict__ out) {
    __shared__ float T[32][33];
    const CzInst in = inst[blockIdx.z];
    const int nd = in.nd, ndp = in.ndp;
    if ((int)blockIdx.x * 32 >= ndp || (int)blockIdx.y * 32 >= ndp) return;
    A += in.a0;
    out += in.a0;
    s += in.agg0 * M;
    const int bi = blockIdx.y, bj = blockIdx.x, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const bool low = bj <= bi;
    for (int r = ty; r < 32; r += 8)
        T[r][tx] = low ? A[(size_t)(bi * 32 + r) * ndp + bj * 32 + tx] : A[(size_t)(bj * 32 + r) * ndp + bi * 32 + tx];
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int i = bi * 32 + r, j = bj * 32 + tx;
        const float v = low && !(bi == bj && tx > r) ? T[r][tx] : T[tx][r];
        out[(size_t)i * ndp + j] = (i < nd && j < nd) ? -v * s[i] * s[j] : 0.f;
    }
}

// ---------------------------------------------------------------------------
// Plan, once per pattern: support points, boxes, row lists

// support point of every DOF object: vertices, midpoints of the edges (the
// sum of two numbers does not depend on their order, so elements that share
// an edge write the same bits), the centre of a quadrilateral
__global__ void k_cz_points(int shape, int ngeom, int nfun, int64_t nelem, const int32_t* __restrict__ conn,
                            const int32_t* __restrict__ edof, const double* __restrict__ X, int D, double* __restrict__ P) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nelem) return;
    const int tetE[6][2] = {{0, 1}, {1, 2}, {2, 0}, {3, 0}, {3, 1}, {3, 2}};
    for (int f = 0; f < nfun; ++f) {
        const int64_t o = edof[(int64_t)f * nelem + e];
        for (int d = 0; d < D; ++d) {
            double v;
            if (f < ngeom) v = X[(int64_t)conn[(int64_t)f * nelem + e] * D + d];
            else if (shape == ISL_QUAD && f == 8) {
                v = 0.0;
                for (int k = 0; k < 4; ++k) v += 0.25 * X[(int64_t)conn[(int64_t)k * nelem + e] * D + d];
            } else {
                const int q = f - ngeom;
                const int a = shape == ISL_QUAD ? q : tetE[q][0], b = shape == ISL_QUAD ? (q + 1) % 4 : tetE[q][1];
                v = 0.5 * (X[(int64_t)conn[(int64_t)a * nelem + e] * D + d] + X[(int64_t)conn[(int64_t)b * nelem + e] * D + d]);
            }
            P[o * D + d] = v;
        }
    }
}

__global__ void k_cz_eqrow(int n3, const int* __restrict__ aeq, int* __restrict__ eqrow) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n3 && aeq[t] >= 0) eqrow[aeq[t]] = t / 3;
}

// point (w: the component, NC = 1, or the mask of constrained components) of every
// row, relative to a vertex of its instance: rounded to FP32 as they stand, the
// points of a mesh far from the origin would coincide
template <int NC>
__global__ void k_cz_rowpts(int64_t ndo, int ncomp, const int32_t* __restrict__ eq, const int* __restrict__ eqrow, int D,
                            const double* __restrict__ P, const CzInst* __restrict__ inst, int ninst,
                            const int32_t* __restrict__ conn, const double* __restrict__ X, float4* __restrict__ xr) {
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= ndo) return;
    auto point = [&](int row) {
        const double* org = X + (size_t)D * conn[inst[ninst > 1 ? inst_of(inst, ninst, row) : 0].elem0];
        return make_float4((float)(P[o * D] - org[0]), (float)(P[o * D + 1] - org[1]), D == 3 ? (float)(P[o * D + 2] - org[2]) : 0.f, 0.f);
    };
    if (NC == 1) {
        for (int c = 0; c < ncomp; ++c) {
            const int e = eq[o * ncomp + c];
            if (e < 0) continue;
            float4 v = point(e);
            v.w = __int_as_float(c);
            xr[e] = v;
        }
    } else {
        int first = -1, mask = 0;
        for (int c = 0; c < 3; ++c) {
            const int e = eq[o * 3 + c];
            if (e < 0) mask |= 1 << c;
            else if (first < 0) first = e;
        }
        if (first < 0) return;
        const int row = eqrow ? eqrow[first] : first / 3;
        float4 v = point(row);
        v.w = __int_as_float(mask);
        xr[row] = v;
    }
}

__device__ inline unsigned f_order(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : b | 0x80000000u;
}
inline float f_unorder(unsigned u) {
    union { unsigned u; float f; } c;
    c.u = (u & 0x80000000u) ? u & 0x7fffffffu : ~u;
    return c.f;
}

__global__ void k_cz_bounds(int n, int ninst, const CzInst* __restrict__ inst, const float4* __restrict__ xr, unsigned* __restrict__ mm) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v[3] = {xr[i].x, xr[i].y, xr[i].z};
        if (ninst > 1) {
            unsigned* o = mm + 6 * inst_of(inst, ninst, i);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const unsigned u = f_order(v[d]);
                if (u < *(volatile unsigned*)(o + d)) atomicMin(o + d, u);
                if (u > *(volatile unsigned*)(o + 3 + d)) atomicMax(o + 3 + d, u);
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) { lo[d] = fminf(lo[d], v[d]); hi[d] = fmaxf(hi[d], v[d]); }
    }
    if (ninst > 1) return;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
        if ((threadIdx.x & 31) == 0) { atomicMin(mm + d, f_order(lo[d])); atomicMax(mm + 3 + d, f_order(hi[d])); }
    }
}

struct Box3 { float lo[3], inv[3]; int m[3], base; };  // m: boxes per direction, base: the instance's first box

__device__ inline int bin_of(const Box3& b, int d, float x) {
    return min(NBIN - 1, max(0, (int)((x - b.lo[d]) * b.inv[d])));
}

// rows per bin, axis and instance
__global__ void k_cz_hist(int n, int ninst, const CzInst* __restrict__ inst, const Box3* __restrict__ box,
                          const float4* __restrict__ xr, int* __restrict__ hist) {
    __shared__ int h[3 * NBIN];
    if (ninst > 1) {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const int k = inst_of(inst, ninst, i);
            const Box3 b = box[k];
            const float v[3] = {xr[i].x, xr[i].y, xr[i].z};
#pragma unroll
            for (int d = 0; d < 3; ++d) atomicAdd(&hist[((size_t)k * 3 + d) * NBIN + bin_of(b, d, v[d])], 1);
        }
        return;
    }
    const Box3 b = box[0];
    for (int k = threadIdx.x; k < 3 * NBIN; k += blockDim.x) h[k] = 0;
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v[3] = {xr[i].x, xr[i].y, xr[i].z};
#pragma unroll
        for (int d = 0; d < 3; ++d) atomicAdd(&h[d * NBIN + bin_of(b, d, v[d])], 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 3 * NBIN; k += blockDim.x)
        if (h[k]) atomicAdd(&hist[k], h[k]);
}

// raw key of every row: (box, component) and sub-box; cut[instance][d][bin] is
// the half-box index along d
template <int NC, int NW>
__global__ void k_cz_key(int n, int ninst, const CzInst* __restrict__ inst, const Box3* __restrict__ box,
                         const unsigned short* __restrict__ cut, int ncomp, const float4* __restrict__ xr, int* __restrict__ key,
                         int* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = ninst > 1 ? inst_of(inst, ninst, i) : 0;
        const Box3 b = box[k];
        const unsigned short* q = cut + (size_t)k * 3 * NBIN;
        const float4 v = xr[i];
        const int h0 = q[bin_of(b, 0, v.x)], h1 = q[NBIN + bin_of(b, 1, v.y)], h2 = q[2 * NBIN + bin_of(b, 2, v.z)];
        int g = ((h2 >> 1) * b.m[1] + (h1 >> 1)) * b.m[0] + (h0 >> 1);
        if (NC == 1) g = g * ncomp + __float_as_int(v.w);
        g += b.base;
        const int s = (h0 & 1) | (h1 & 1) << 1 | (NW == 8 ? (h2 & 1) << 2 : 0);
        key[i] = g * NW + s;
        atomicAdd(&cnt[g * NW + s], 1);
    }
}

// sort key of every row: sub-aggregate, then (scalar rows) the length, falling
// and rising in turn, so that the slices of the aggregate-ordered copy need
// little padding inside a sub-aggregate and across two
constexpr int LEN_BITS = 10;
template <int NC, int NW>
__global__ void k_cz_rekey(int n, const int* __restrict__ map, const int* __restrict__ rowptr, int* __restrict__ key,
                           int* __restrict__ row) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = key[i], top = (1 << LEN_BITS) - 1;
        const int sub = map[k / NW] * NW + k % NW;
        const int len = NC == 1 ? min(top, rowptr[i + 1] - rowptr[i]) : 0;
        key[i] = sub << LEN_BITS | (sub & 1 ? len : top - len);
        row[i] = i;
    }
}

// centre and rms radius of every aggregate, then the rows' scaled positions
template <int NC, int NW>
__global__ void __launch_bounds__(NW * 32) k_cz_nodes(const int* __restrict__ sofs, const int* __restrict__ list,
                                                      const int* __restrict__ key, const float4* __restrict__ xr,
                                                      float4* __restrict__ lnode, float4* __restrict__ yrow,
                                                      int* __restrict__ pos) {
    __shared__ double sh[32];
    __shared__ double cen[3], irad;
    const int t0 = sofs[blockIdx.x * NW], t1 = sofs[(blockIdx.x + 1) * NW];
    double s[3] = {0.0, 0.0, 0.0};
    for (int t = t0 + threadIdx.x; t < t1; t += NW * 32) {
        const float4 v = xr[list[t]];
        s[0] += v.x; s[1] += v.y; s[2] += v.z;
    }
    for (int d = 0; d < 3; ++d) {
        const double v = block_sum(s[d], sh);
        if (threadIdx.x == 0) cen[d] = v / (t1 - t0);
    }
    __syncthreads();
    double q = 0.0;
    for (int t = t0 + threadIdx.x; t < t1; t += NW * 32) {
        const float4 v = xr[list[t]];
        const double a = v.x - cen[0], b = v.y - cen[1], c = v.z - cen[2];
        q += a * a + b * b + c * c;
    }
    const double qq = block_sum(q, sh);
    if (threadIdx.x == 0) irad = qq > 0.0 ? 1.0 / sqrt(qq / (t1 - t0)) : 0.0;
    __syncthreads();
    for (int t = t0 + threadIdx.x; t < t1; t += NW * 32) {
        const int row = list[t];
        const float4 v = xr[row];
        float4 y = make_float4((float)((v.x - cen[0]) * irad), (float)((v.y - cen[1]) * irad), (float)((v.z - cen[2]) * irad), 0.f);
        y.w = __int_as_float(NC == 3 ? row | __float_as_int(v.w) << ROW_BITS : t);
        lnode[t] = y;
        y.w = __int_as_float(key[t] >> LEN_BITS);
        yrow[NC == 3 ? row : t] = y;
        pos[row] = t;
    }
}

// Allocations of the plan.  One that fails leaves the system to the one-level
// solve (coarse_drop); the test hook makes the n-th one fail.
template <typename T>
cudaError_t cz_alloc(isl_ctx* c, DBuf<T>& b, size_t count) {
    if (c->alloc_test > 0 && --c->alloc_test == 0) return cudaErrorMemoryAllocation;
    return b.alloc(count);
}
#define CZ_ALLOC(c, b, count) ISL_CHECK_CUDA(c, cz_alloc(c, b, count))
// declared after the scratch buffers of a function, so that these are given
// back after the kernels that use them, on every way out
struct StreamDone {
    cudaStream_t st;
    ~StreamDone() { cudaStreamSynchronize(st); }
};

unsigned grid_for(const isl_ctx* c, int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8LL * c->sm_count)); }

// Boxes per direction of one instance: near-cubic boxes of edge h, which gives
// the target number of them over the directions that are at least one edge
// long; then the largest product of rounded-down or rounded-up counts within it.
void choose_boxes(int D, const double* L, int target, int* mbox) {
    const double Lmax = std::max(L[0], std::max(L[1], L[2]));
    bool use[3] = {L[0] > 0.0, L[1] > 0.0, L[2] > 0.0};
    mbox[0] = mbox[1] = mbox[2] = 1;
    if (!(Lmax > 0.0)) return;
    double h = Lmax;
    for (bool again = true; again;) {
        double vol = 1.0;
        int nd = 0;
        for (int d = 0; d < D; ++d)
            if (use[d]) { vol *= L[d]; ++nd; }
        h = std::pow(vol / target, 1.0 / nd);
        again = false;
        for (int d = 0; d < D; ++d)
            if (use[d] && nd > 1 && L[d] < h) { use[d] = false; again = true; break; }
    }
    int64_t best = 0;
    for (int pick = 0; pick < 1 << D; ++pick) {
        int64_t tot = 1;
        int m[3] = {1, 1, 1};
        for (int d = 0; d < D; ++d) {
            m[d] = use[d] ? std::max(1, (int)std::min(L[d] / h, (double)target) + ((pick >> d) & 1)) : 1;
            tot *= m[d];
        }
        if (tot <= target && tot > best) {
            best = tot;
            for (int d = 0; d < 3; ++d) mbox[d] = m[d];
        }
    }
}

template <int NC, int M, int NW>
int build_plan(isl_ctx* c, CzPlan& z) {
    cudaStream_t st = c->stream;
    const int D = c->dim, n = (int)z.nrow, ni = (int)c->ninst;
    z.ninst = ni;
    z.hinst.assign((size_t)ni, CzInst{});
    for (int k = 0; k < ni; ++k) {
        z.hinst[k].row0 = ni > 1 ? (int)c->inst_eq_off[k] : 0;
        z.hinst[k].nrow = ni > 1 ? (int)(c->inst_eq_off[k + 1] - c->inst_eq_off[k]) : n;
        z.hinst[k].elem0 = ni > 1 ? (int)c->inst_elem_off[k] : 0;
    }
    DBuf<double> P;
    DBuf<float4> xr;
    DBuf<int32_t> eqrow, hist, key, key2, row, cnt, map;
    DBuf<unsigned> mm;
    DBuf<unsigned short> dcut;
    DBuf<Box3> dbox;
    DBuf<char> tmp;
    StreamDone done{st};
    std::vector<unsigned> hmm((size_t)6 * ni, 0u);
    for (int k = 0; k < ni; ++k)
        for (int d = 0; d < 3; ++d) hmm[6 * k + d] = 0xffffffffu;
    CZ_ALLOC(c, P, (size_t)c->ndofobj * D);
    CZ_ALLOC(c, xr, n);
    CZ_ALLOC(c, mm, hmm.size());
    CZ_ALLOC(c, hist, (size_t)3 * NBIN * ni);
    CZ_ALLOC(c, z.inst, ni);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(mm.p, hmm.data(), hmm.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.inst.p, z.hinst.data(), (size_t)ni * sizeof(CzInst), cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(hist.p, 0, (size_t)3 * NBIN * ni * 4, st));
    k_cz_points<<<(unsigned)((c->nelem + 255) / 256), 256, 0, st>>>(c->shape, c->ngeom, c->nfun, c->nelem, c->dconn.p,
                                                                     c->dedof.p, c->dX.p, D, P.p);
    if (NC == 3 && c->bpad) {
        CZ_ALLOC(c, eqrow, (size_t)c->neq);
        k_cz_eqrow<<<(3 * n + 255) / 256, 256, 0, st>>>(3 * n, c->dbaeq.p, eqrow.p);
        c->launches += 1;
    }
    k_cz_rowpts<NC><<<(unsigned)((c->ndofobj + 255) / 256), 256, 0, st>>>(c->ndofobj, c->ncomp, c->deq.p, eqrow.p, D, P.p, z.inst.p, ni,
                                                                                    c->dconn.p, c->dX.p, xr.p);
    const unsigned g = grid_for(c, n);
    k_cz_bounds<<<g, 256, 0, st>>>(n, ni, z.inst.p, xr.p, mm.p);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hmm.data(), mm.p, hmm.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    const int comps = NC == 1 ? c->ncomp : 1;
    std::vector<Box3> box((size_t)ni);
    int64_t nbox = 0;
    for (int k = 0; k < ni; ++k) {
        Box3& b = box[k];
        double L[3] = {0, 0, 0};
        for (int d = 0; d < 3; ++d) {
            const float lo = f_unorder(hmm[6 * k + d]), hi = f_unorder(hmm[6 * k + 3 + d]);
            L[d] = d < D && z.hinst[k].nrow ? (double)hi - lo : 0.0;
            if (!(L[d] >= 0.0) || !std::isfinite(L[d])) return ISL_OK;  // no usable coordinates: one-level
            b.lo[d] = z.hinst[k].nrow ? lo : 0.f;
            b.inv[d] = L[d] > 0.0 ? (float)(NBIN / L[d]) : 0.f;
        }
        choose_boxes(D, L, std::max(1, coarse_target(z.hinst[k].nrow) / comps), b.m);
        b.base = (int)nbox;
        nbox += (int64_t)b.m[0] * b.m[1] * b.m[2] * comps;
    }
    if (nbox * NW >= (int64_t)1 << (31 - LEN_BITS) || ni > 65535) return ISL_OK;  // sort keys, launch grids
    CZ_ALLOC(c, dbox, ni);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(dbox.p, box.data(), (size_t)ni * sizeof(Box3), cudaMemcpyHostToDevice, st));
    k_cz_hist<<<ni > 1 ? g : std::min(g, (unsigned)c->sm_count), 256, 0, st>>>(n, ni, z.inst.p, dbox.p, xr.p, hist.p);
    std::vector<int32_t> hh((size_t)3 * NBIN * ni);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hh.data(), hist.p, hh.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    // cuts at the quantiles of the rows, two half-boxes per box
    std::vector<unsigned short> cut((size_t)3 * NBIN * ni, 0);
    for (int k = 0; k < ni; ++k)
        for (int d = 0; d < D; ++d) {
            const int64_t parts = 2 * box[k].m[d];
            int64_t run = 0;
            for (int b = 0; b < NBIN; ++b) {
                const size_t i = ((size_t)k * 3 + d) * NBIN + b;
                cut[i] = (unsigned short)std::min<int64_t>(parts - 1, (run + hh[i] / 2) * parts / std::max(z.hinst[k].nrow, 1));
                run += hh[i];
            }
        }
    CZ_ALLOC(c, dcut, cut.size());
    CZ_ALLOC(c, key, n);
    CZ_ALLOC(c, key2, n);
    CZ_ALLOC(c, row, n);
    CZ_ALLOC(c, z.perm, n);
    CZ_ALLOC(c, z.pos, n);
    CZ_ALLOC(c, cnt, (size_t)nbox * NW);
    CZ_ALLOC(c, map, nbox);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(dcut.p, cut.data(), cut.size() * 2, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(cnt.p, 0, (size_t)nbox * NW * 4, st));
    k_cz_key<NC, NW><<<g, 256, 0, st>>>(n, ni, z.inst.p, dbox.p, dcut.p, c->ncomp, xr.p, key.p, cnt.p);
    std::vector<int32_t> hc((size_t)nbox * NW), hmap((size_t)nbox, -1), so, ai;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hc.data(), cnt.p, hc.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    // the boxes that hold rows, per instance
    int32_t run = 0, na = 0;
    long long a0 = 0, p0 = 0;
    int rc0 = 0;
    for (int k = 0; k < ni; ++k) {
        CzInst& in = z.hinst[k];
        in.agg0 = na;
        const int64_t end = k + 1 < ni ? box[k + 1].base : nbox;
        for (int64_t b = box[k].base; b < end; ++b) {
            int32_t tot = 0;
            for (int s = 0; s < NW; ++s) tot += hc[(size_t)b * NW + s];
            if (!tot) continue;
            hmap[(size_t)b] = na++;
            ai.push_back(k);
            for (int s = 0; s < NW; ++s) { so.push_back(run); run += hc[(size_t)b * NW + s]; }
        }
        in.nagg = na - in.agg0;
        in.nd = in.nagg * M;
        in.ndp = std::max(1, (in.nd + TB - 1) / TB) * TB;
        in.a0 = a0;
        in.p0 = p0;
        in.rc0 = rc0;
        a0 += (long long)in.ndp * in.ndp;
        p0 += 2LL * TB * in.ndp + 2 * TB * TB;
        rc0 += 2 * in.ndp;
    }
    so.push_back(run);
    z.nagg = na;
    z.nd = z.hinst[0].nd;
    z.ndp = z.hinst[0].ndp;
    if (na == 0) return ISL_OK;
    CZ_ALLOC(c, z.sofs, so.size());
    CZ_ALLOC(c, z.agg_inst, ai.size());
    CZ_ALLOC(c, z.lnode, n);
    CZ_ALLOC(c, z.yrow, n);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.inst.p, z.hinst.data(), (size_t)ni * sizeof(CzInst), cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.sofs.p, so.data(), so.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.agg_inst.p, ai.data(), ai.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(map.p, hmap.data(), hmap.size() * 4, cudaMemcpyHostToDevice, st));
    k_cz_rekey<NC, NW><<<g, 256, 0, st>>>(n, map.p, c->drowptr.p, key.p, row.p);
    int bits = 1;
    while ((1 << bits) < na * NW) ++bits;
    bits += LEN_BITS;
    size_t tb = 0;
    ISL_CHECK_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, tb, key.p, key2.p, row.p, z.perm.p, n, 0, bits, st));
    CZ_ALLOC(c, tmp, std::max<size_t>(tb, 1));
    ISL_CHECK_CUDA(c, cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.p, key2.p, row.p, z.perm.p, n, 0, bits, st));
    k_cz_nodes<NC, NW><<<na, NW * 32, 0, st>>>(z.sofs.p, z.perm.p, key2.p, xr.p, z.lnode.p, z.yrow.p, z.pos.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    CZ_ALLOC(c, z.dsub, (size_t)na * NW * M * M);
    CZ_ALLOC(c, z.dagg, (size_t)na * M * M);
    CZ_ALLOC(c, z.scale, (size_t)na * M);
    CZ_ALLOC(c, z.rc, rc0);
    CZ_ALLOC(c, z.acc, (size_t)a0);
    CZ_ALLOC(c, z.a, (size_t)a0);
    CZ_ALLOC(c, z.ainv, (size_t)a0);
    CZ_ALLOC(c, z.panel, (size_t)p0);
    CZ_ALLOC(c, z.amax, na + ni);
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.rc.p, 0, (size_t)rc0 * 4, st));  // the padding stays zero
    c->launches += 10;
    z.hsofs = std::move(so);
    z.ok = true;
    return ISL_OK;
}

// Aggregate-ordered copies of the matrix (t-space: the order of the row list).
// The update and coarse kernels then read their vectors contiguously, and the
// rows of a slice gather from a few neighbouring boxes.

// scalar rows: row lengths of a slice
__global__ void k_pz_width(int n, int nslice, const int* __restrict__ perm, const int* __restrict__ rowptr, int* __restrict__ wid) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nslice) return;
    int w = 0;
    for (int t = s * 32; t < min(n, s * 32 + 32); ++t) w = max(w, rowptr[perm[t] + 1] - rowptr[perm[t]]);
    wid[s] = w;
}
__global__ void k_pz_cols(int n, int nslice, const int* __restrict__ perm, const int* __restrict__ pos, const int* __restrict__ rowptr,
                          const int* __restrict__ colind, const int* __restrict__ soff, const int* __restrict__ swid,
                          int* __restrict__ col, short* __restrict__ col16, int* __restrict__ far) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nslice * 32) return;
    const int row = t < n ? perm[t] : -1, base = t < n ? t : 0;
    const int lo = row >= 0 ? rowptr[row] : 0, len = row >= 0 ? rowptr[row + 1] - lo : 0;
    const int o = soff[t >> 5] + (t & 31), w = swid[t >> 5];
    for (int k = 0; k < w; ++k) {
        const int j = k < len ? pos[colind[lo + k]] : base, d = j - base;
        col[o + 32 * k] = j;
        if (d < -32767 || d > 32767) atomicOr(far, 1);
        col16[o + 32 * k] = (short)d;
    }
}
// values: the loads of a lane run along its CSR row
__global__ void k_pz_values(int n, const int* __restrict__ perm, const int* __restrict__ rowptr, const float* __restrict__ val,
                            const int* __restrict__ soff, float* __restrict__ sv) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int lo = rowptr[perm[t]], hi = rowptr[perm[t] + 1], o = soff[t >> 5] + (t & 31);
        for (int k = lo; k < hi; ++k) sv[o + 32 * (k - lo)] = val[k];
    }
}
__global__ void k_pz_dinv(int n, const int* __restrict__ perm, const int* __restrict__ diag, const float* __restrict__ val,
                          float* __restrict__ dinv) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const float d = val[diag[perm[t]]];
        dinv[t] = d != 0.f ? 1.f / d : 1.f;
    }
}

// row lists for the one-cluster solve: (block) CSR in t-space
__global__ void k_pz_len(int n, const int* __restrict__ perm, const int* __restrict__ ptr, int* __restrict__ len) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t <= n) len[t] = t < n ? ptr[perm[t] + 1] - ptr[perm[t]] : 0;
}
__global__ void k_pz_csr_cols(int n, const int* __restrict__ perm, const int* __restrict__ pos, const int* __restrict__ ptr,
                              const int* __restrict__ colind, const int* __restrict__ rp, int* __restrict__ col) {
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < n; t += gridDim.x * 8) {
        const int lo = ptr[perm[t]], len = rp[t + 1] - rp[t];
        for (int k = threadIdx.x & 31; k < len; k += 32) col[rp[t] + k] = pos[colind[lo + k]];
    }
}
// node blocks: inverse diagonal blocks in list order, [9][n]
__global__ void k_pz_binv(int n, const int* __restrict__ perm, const float* __restrict__ binv, float* __restrict__ dinv) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
        for (int k = 0; k < 9; ++k) dinv[(size_t)k * n + t] = binv[(size_t)9 * perm[t] + k];
}
template <int NC>
__global__ void k_pz_csr_values(int n, const int* __restrict__ perm, const int* __restrict__ ptr, const int* __restrict__ sdst,
                                const float* __restrict__ src, const int* __restrict__ rp, int nblk, float* __restrict__ val) {
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < n; t += gridDim.x * 8) {
        const int lo = ptr[perm[t]], len = rp[t + 1] - rp[t];
        for (int k = threadIdx.x & 31; k < len; k += 32) {
            if (NC == 1) {
                val[rp[t] + k] = src[lo + k];
            } else {
                const int slot = sdst[lo + k];
                const float* g = src + (size_t)(slot >> 5) * 288 + (slot & 31);
#pragma unroll
                for (int e = 0; e < 9; ++e) val[(size_t)e * nblk + rp[t] + k] = g[32 * e];
            }
        }
    }
}

// shared memory of the one-launch solve; *ms, *as: the matrix and the rows of
// the inverse fit too (in that order)
constexpr size_t CLU_SMEM_MAX = 224 * 1024;
constexpr int CLS_ENT = 8192;  // stored entries a CTA of a batch's cluster takes, about
size_t cluster_need(const CzPlan& z, int rows, int aggs, int ndp, int ent, bool m, bool s) {
    return z.nc == 3 ? clu_smem<3, 6, 8>(rows, aggs, ndp, ent, m, s)
           : z.m == 4 ? clu_smem<1, 4, 8>(rows, aggs, ndp, ent, m, s) : clu_smem<1, 3, 4>(rows, aggs, ndp, ent, m, s);
}
size_t cluster_smem(const CzClass& k, bool* ms, bool* as) {
    const auto& need = k.smem;
    *ms = need[1][0] <= CLU_SMEM_MAX;
    *as = need[*ms][1] <= CLU_SMEM_MAX;
    return need[*ms][*as];
}

inline size_t cluster_smem_min(const CzClass& k) { return k.smem[0][0]; }

// columns of the aggregate-ordered sliced-ELL copy (scalar systems), once per pattern
int build_sell(isl_ctx* c, CzPlan& z) {
    if (z.sell_built) return ISL_OK;
    cudaStream_t st = c->stream;
    const int n = (int)z.nrow, ns = (n + 31) / 32;
    CZ_ALLOC(c, z.swid, ns);
    CZ_ALLOC(c, z.soff, ns + 1);
    k_pz_width<<<(ns + 127) / 128, 128, 0, st>>>(n, ns, z.perm.p, c->drowptr.p, z.swid.p);
    std::vector<int32_t> wid(ns), off(ns + 1);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(wid.data(), z.swid.p, (size_t)ns * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    int64_t tot = 0;
    for (int s = 0; s < ns; ++s) {
        off[s] = (int32_t)tot;
        tot += 32LL * wid[s];
        if (tot >= INT32_MAX) { z.ok = false; return ISL_OK; }
    }
    off[ns] = (int32_t)tot;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.soff.p, off.data(), (size_t)(ns + 1) * 4, cudaMemcpyHostToDevice, st));
    CZ_ALLOC(c, z.col, tot);
    CZ_ALLOC(c, z.col16, tot);
    CZ_ALLOC(c, z.val, tot);
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.val.p, 0, (size_t)tot * 4, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->dflags.p + 1, 0, sizeof(int), st));
    k_pz_cols<<<(ns * 32 + 255) / 256, 256, 0, st>>>(n, ns, z.perm.p, z.pos.p, c->drowptr.p, c->dcolind.p, z.soff.p, z.swid.p,
                                                      z.col.p, z.col16.p, c->dflags.p + 1);
    int far = 0;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(&far, c->dflags.p + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    z.short_cols = far == 0;
    if (far) z.col16.release();
    z.nslice = ns;
    c->launches += 2;
    z.sell_built = true;
    return ISL_OK;
}

// (block) CSR in t-space for the one-cluster solve, once per pattern
int build_csr(isl_ctx* c, CzPlan& z) {
    const bool batch = c->ninst > 1 || c->force_batched;
    if (z.csr_built && z.batch == batch) return ISL_OK;
    z.csr_built = false;
    z.batch = batch;
    cudaStream_t st = c->stream;
    const int n = (int)z.nrow;
    const int* ptr = z.nc == 3 ? c->dbptr.p : c->drowptr.p;
    z.nent = z.nc == 3 ? c->nblk : c->nnz;
    DBuf<int32_t> len;
    DBuf<char> tmp;
    StreamDone done{st};
    CZ_ALLOC(c, len, n + 1);
    CZ_ALLOC(c, z.rp, n + 1);
    CZ_ALLOC(c, z.ci, z.nent);
    CZ_ALLOC(c, z.cv, (size_t)z.nc * z.nc * z.nent);
    k_pz_len<<<n / 256 + 1, 256, 0, st>>>(n, z.perm.p, ptr, len.p);
    size_t tb = 0;
    ISL_CHECK_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tb, len.p, z.rp.p, n + 1, st));
    CZ_ALLOC(c, tmp, std::max<size_t>(tb, 1));
    ISL_CHECK_CUDA(c, cub::DeviceScan::ExclusiveSum(tmp.p, tb, len.p, z.rp.p, n + 1, st));
    k_pz_csr_cols<<<(n + 7) / 8, 256, 0, st>>>(n, z.perm.p, z.pos.p, ptr, z.nc == 3 ? c->dbcol.p : c->dcolind.p, z.rp.p, z.ci.p);
    std::vector<int32_t> rp(n + 1);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(rp.data(), z.rp.p, (size_t)(n + 1) * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    // per instance: contiguous aggregates per CTA, balanced by stored entries
    const int nw = z.m == 3 ? 4 : 8;
    const size_t nc1 = (size_t)z.ncta + 1;
    z.hcta.assign(nc1 * z.ninst, 0);
    std::vector<int32_t> order, big_cta;
    auto split = [&](CzInst& in, int ncta, int32_t* cta) {
        in.rows = in.aggs = in.ent = 0;
        const int64_t e0 = rp[in.row0], ent = rp[in.row0 + in.nrow] - e0;
        int ag = in.agg0;
        cta[0] = ag;
        for (int k = 0; k < ncta; ++k) {
            const int from = ag, end = in.agg0 + in.nagg;
            const int64_t goal = 2 * (e0 + ent * (k + 1) / ncta);
            while (ag < end && (k == ncta - 1 ||
                                (int64_t)rp[z.hsofs[(size_t)ag * nw]] + rp[z.hsofs[(size_t)(ag + 1) * nw]] < goal)) ++ag;
            cta[k + 1] = ag;
            const int t0 = z.hsofs[(size_t)from * nw], t1 = z.hsofs[(size_t)ag * nw];
            in.rows = std::max(in.rows, t1 - t0);
            in.aggs = std::max(in.aggs, ag - from);
            in.ent = std::max(in.ent, rp[t1] - rp[t0]);
        }
        return cluster_need(z, in.rows, in.aggs, in.ndp, in.ent, false, false) <= CLU_SMEM_MAX;
    };
    // an instance lays its shared memory out for itself: a launch takes what the
    // largest of its instances needs, and none is sized by the shares of two
    auto admit = [&](const CzInst& in, CzClass& cl) {
        cl.count += 1;
        for (int k = 0; k < 4; ++k) {
            size_t& need = cl.smem[k >> 1][k & 1];
            need = std::max(need, cluster_need(z, in.rows, in.aggs, in.ndp, in.ent, k >> 1, k & 1));
        }
    };
    z.big.clear();
    z.cls.clear();
    z.big_ncta = c->sm_count;
    z.big_cls = {};
    // In a batch a cluster has as few CTAs as give each at most CLS_ENT entries
    // (and enough for them to fit), whatever the other instances: a small one
    // waits for fewer peers, and more run at once.  600 Q1 instances to 1e-10 with 16
    // CTAs each / so / one-level: side 4 10.4 / 0.76 / 2.1 ms, side 32 29.1 / 3.8 /
    // 7.7 ms; with half as many entries to a CTA the latter takes 6.4 ms, and 150 P2
    // meshes of 5^3 cells 3.6 ms instead of 2.2.  (Four of side 32 alone: 0.45 / 0.55 ms.)
    std::vector<std::vector<int32_t>> by_size;  // by the cluster's CTAs: 1, 2, 4, ... ncta
    for (int k = 1; k < z.ncta; k *= 2) by_size.push_back({});
    by_size.push_back({});
    for (int i = 0; i < z.ninst; ++i) {
        CzInst& in = z.hinst[i];
        int32_t* cta = &z.hcta[nc1 * i];
        int cl = batch ? 0 : (int)by_size.size() - 1;
        auto ctas = [&] { return std::min(1 << cl, z.ncta); };
        while (cl + 1 < (int)by_size.size() && (int64_t)ctas() * CLS_ENT < rp[in.row0 + in.nrow] - rp[in.row0]) ++cl;
        while (!split(in, ctas(), cta) && cl + 1 < (int)by_size.size()) ++cl;
        if (cluster_need(z, in.rows, in.aggs, in.ndp, in.ent, false, false) > CLU_SMEM_MAX && z.ninst > 1) {
            std::vector<int32_t> cb((size_t)z.big_ncta + 1);
            if (!split(in, z.big_ncta, cb.data())) continue;  // one-level
            z.big.push_back(i);
            big_cta.insert(big_cta.end(), cb.begin(), cb.end());
            admit(in, z.big_cls);
            continue;
        }
        by_size[(size_t)cl].push_back(i);
    }
    for (int k = (int)by_size.size() - 1; k >= 0; --k) {
        std::vector<int32_t>& v = by_size[(size_t)k];
        if (v.empty()) continue;
        std::stable_sort(v.begin(), v.end(), [&](int32_t a, int32_t b) { return z.hinst[a].nrow > z.hinst[b].nrow; });
        CzClass cl = {k + 1 == (int)by_size.size() ? z.ncta : 1 << k, (int)order.size(), 0, {}};
        for (const int32_t i : v) admit(z.hinst[i], cl);
        order.insert(order.end(), v.begin(), v.end());
        z.cls.push_back(cl);
    }
    if (batch && z.ninst == 1 && cluster_smem_min(z.cls[0]) > CLU_SMEM_MAX) z.cls.clear();
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.inst.p, z.hinst.data(), (size_t)z.ninst * sizeof(CzInst), cudaMemcpyHostToDevice, st));
    if (!z.big.empty()) {
        CZ_ALLOC(c, z.cta_big, big_cta.size());
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.cta_big.p, big_cta.data(), big_cta.size() * 4, cudaMemcpyHostToDevice, st));
        ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    }
    if (z.ninst > 1 && !order.empty()) {
        CZ_ALLOC(c, z.order, order.size());
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.order.p, order.data(), order.size() * 4, cudaMemcpyHostToDevice, st));
    }
    CZ_ALLOC(c, z.cta, z.hcta.size());
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.cta.p, z.hcta.data(), z.hcta.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    c->launches += 3;
    z.csr_built = true;
    return ISL_OK;
}

template <int NC, int M, int NW>
int numeric(isl_ctx* c, CzPlan& z, const CzMat& A) {
    cudaStream_t st = c->stream;
    int ndp = 0;
    for (const CzInst& in : z.hinst) ndp = std::max(ndp, in.ndp);
    const int nt = ndp / TB, ni = z.ninst;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.acc.p, 0, z.acc.n * 8, st));
    const int* aeq = NC == 3 && c->bpad ? c->dbaeq.p : nullptr;
    float* top = z.amax.p + z.nagg;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.amax.p, 0, z.amax.n * 4, st));
    const dim3 gmax(z.nagg, 4);
    if (c->have64) k_cz_amax<NC, NW><<<gmax, NW * 32, 0, st>>>(z.sofs.p, z.perm.p, aeq, c->ddiag.p, c->dval64.p, z.agg_inst.p, z.amax.p, top);
    else k_cz_amax<NC, NW><<<gmax, NW * 32, 0, st>>>(z.sofs.p, z.perm.p, aeq, c->ddiag.p, c->dval32.p, z.agg_inst.p, z.amax.p, top);
    k_cz_galerkin<NC, M, NW><<<z.nagg, NW * 32, 0, st>>>(A, z.lnode.p, z.yrow.p, z.sofs.p, z.inst.p, z.agg_inst.p, z.amax.p, top,
                                                         z.acc.p, z.dsub.p, z.dagg.p);
    k_cz_sub_inv<M><<<(z.nagg * NW + 63) / 64, 64, 0, st>>>(z.nagg * NW, z.dsub.p);
    k_cz_scale<M><<<(z.nagg + 127) / 128, 128, 0, st>>>(z.nagg, z.dagg.p, z.scale.p);
    const dim3 g32(ndp / 32, ndp / 32, ni);
    k_cz_form<M><<<g32, 256, 0, st>>>(z.inst.p, z.acc.p, z.dagg.p, z.scale.p, z.amax.p, top, z.a.p);
    ISL_CHECK_CUDA(c, cudaFuncSetAttribute(k_gj_step, cudaFuncAttributeMaxDynamicSharedMemorySize, GJ_SMEM));
    k_gj_first<<<dim3(nt, ni), 256, 0, st>>>(z.inst.p, z.a.p, z.panel.p);
    for (int k = 0; k < nt; ++k) k_gj_step<<<dim3(nt * (nt + 1) / 2, ni), 256, GJ_SMEM, st>>>(z.inst.p, k, z.a.p, z.panel.p);
    k_cz_unscale<M><<<g32, 256, 0, st>>>(z.inst.p, z.a.p, z.scale.p, z.ainv.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 7 + nt;
    return ISL_OK;
}

template <int NC, int M, int NW, int WPS>
void launch_iter_w(const CzPlan& z, cudaStream_t st, const CzIter& a, int mode) {
    const unsigned g = (unsigned)z.nagg, t = NW * WPS * 32;
    if (mode == CZ_UPDATE) {
        // chained: the next kernel is resident with its rows and dense lines on the way
        // when this one ends.  An iteration of 531k scalar rows 58.9 -> 54.7 us (four
        // kernels), of 103k 32.2 -> 30.3.  The product of node blocks is not chained: its
        // gathers would have to leave the read-only path, which costs as much as the launch
        // gains (9,261 nodes 22.3 -> 22.8 us)
        launch_chained(k_cz_update<NC, M, NW, WPS, CZ_UPDATE>, g, t, st, a);
        launch_chained(k_cz_coarse<NC, M, NW, WPS, CZ_UPDATE>, g, t, st, a);
    } else if (mode == CZ_INIT) {
        k_cz_update<NC, M, NW, WPS, CZ_INIT><<<g, t, 0, st>>>(a);
        k_cz_coarse<NC, M, NW, WPS, CZ_INIT><<<g, t, 0, st>>>(a);
    } else {
        k_cz_update<NC, M, NW, WPS, CZ_RESTART><<<g, t, 0, st>>>(a);
        k_cz_coarse<NC, M, NW, WPS, CZ_RESTART><<<g, t, 0, st>>>(a);
    }
}
// warps per sub-aggregate: enough that a lane takes two rows or so
template <int NC, int M, int NW>
void launch_iter(const CzPlan& z, cudaStream_t st, const CzIter& a, int mode) {
    const int64_t per_sub = z.nrow / std::max(1, z.nagg * NW);
    if (per_sub > 48) launch_iter_w<NC, M, NW, 2>(z, st, a, mode);
    else launch_iter_w<NC, M, NW, 1>(z, st, a, mode);
}

}  // namespace

#define CZ_DISPATCH(z, F, ...)                                 \
    ((z).nc == 3 ? F<3, 6, 8>(__VA_ARGS__)                     \
                 : (z).m == 4 ? F<1, 4, 8>(__VA_ARGS__) : F<1, 3, 4>(__VA_ARGS__))

int coarse_plan(isl_ctx* c, int nc, int64_t nrow, int ncta) {
    CzPlan& z = c->cz;
    if (z.serial != c->pattern_serial || z.nc != nc) {
        z.ok = z.sell_built = z.csr_built = false;
        z.num_serial = z.sell_serial = z.csr_serial = z.binv_serial = -1;
        z.spmv_kind = 0;
        z.nc = nc;
        z.m = nc == 3 ? 6 : 1 + c->dim;
        z.nrow = nrow;
        z.serial = c->pattern_serial;
        if (nrow >= (1 << ROW_BITS) || c->fedeg > 2 || (c->fedeg == 2 && c->shape == ISL_HEX) || (c->ninst != 1 && nc != 1)) return ISL_OK;
        const int rc = CZ_DISPATCH(z, build_plan, c, z);
        if (rc != ISL_OK) return rc;
    }
    if (!z.ok) return ISL_OK;
    if (ncta > 0) {
        if (ncta != z.ncta) z.csr_built = false;
        z.ncta = ncta;
        return build_csr(c, z);
    }
    return nc == 1 ? build_sell(c, z) : ISL_OK;
}

void coarse_drop(isl_ctx* c) {
    cudaStreamSynchronize(c->stream);
    cudaGetLastError();
    if (c->cz_exec) cudaGraphExecDestroy(c->cz_exec);
    c->cz_exec = nullptr;
    c->cz_key.clear();
    CzPlan& z = c->cz;
    z.ok = z.sell_built = z.csr_built = false;
    z.bnd_serial = -1;
    for (auto* b : {&z.agg_inst, &z.order, &z.cta_big, &z.sofs, &z.perm, &z.pos, &z.soff, &z.swid, &z.col, &z.bnd, &z.rp, &z.ci, &z.cta}) b->release();
    for (auto* b : {&z.dsub, &z.dagg, &z.scale, &z.rc, &z.a, &z.ainv, &z.panel, &z.binv, &z.val, &z.cv}) b->release();
    z.lnode.release(); z.yrow.release(); z.inst.release(); z.res.release(); z.amax.release(); z.acc.release(); z.col16.release();
}

int coarse_results(isl_ctx* c) {
    CZ_ALLOC(c, c->cz.res, c->ninst);
    ISL_CHECK_CUDA(c, cudaMemsetAsync(c->cz.res.p, 0, (size_t)c->ninst * sizeof(OlScal), c->stream));
    return ISL_OK;
}

int coarse_numeric(isl_ctx* c, bool csr, float* dinv) {
    CzPlan& z = c->cz;
    cudaStream_t st = c->stream;
    const int n = (int)z.nrow;
    CzMat A = {c->dsoff.p, c->dswid.p, nullptr, c->dscol.p, c->dsval.p};
    if (csr && z.csr_serial != c->asm_serial) {
        const unsigned g = (unsigned)std::min<int64_t>((n + 7) / 8, 32LL * c->sm_count);
        if (z.nc == 3) k_pz_csr_values<3><<<g, 256, 0, st>>>(n, z.perm.p, c->dbptr.p, c->dsdst.p, c->dsval.p, z.rp.p, (int)z.nent, z.cv.p);
        else k_pz_csr_values<1><<<g, 256, 0, st>>>(n, z.perm.p, c->drowptr.p, nullptr, c->dval32.p, z.rp.p, (int)z.nent, z.cv.p);
        c->launches += 1;
        z.csr_serial = c->asm_serial;
    }
    if (z.nc == 1) {
        if (!csr && z.sell_serial != c->asm_serial) {
            k_pz_values<<<grid_for(c, n), 256, 0, st>>>(n, z.perm.p, c->drowptr.p, c->dval32.p, z.soff.p, z.val.p);
            c->launches += 1;
            z.sell_serial = c->asm_serial;
        }
        k_pz_dinv<<<grid_for(c, n), 256, 0, st>>>(n, z.perm.p, c->ddiag.p, c->dval32.p, dinv);
        c->launches += 1;
        if (csr) A = {nullptr, nullptr, z.rp.p, z.ci.p, z.cv.p};
        else A = {z.soff.p, z.swid.p, nullptr, z.col.p, z.val.p};
    } else if (!csr && z.binv_serial != c->asm_serial) {
        CZ_ALLOC(c, z.binv, (size_t)9 * n);
        k_pz_binv<<<grid_for(c, n), 256, 0, st>>>(n, z.perm.p, dinv, z.binv.p);
        c->launches += 1;
        z.binv_serial = c->asm_serial;
    }
    ISL_CHECK_CUDA(c, cudaGetLastError());
    if (z.num_serial == c->asm_serial) return ISL_OK;
    const int rc = CZ_DISPATCH(z, numeric, c, z, A);
    if (rc == ISL_OK) z.num_serial = c->asm_serial;
    return rc;
}

// 2: with its matrix on chip, 1: without, 0: not at all
int coarse_cluster_fits(const isl_ctx* c, bool grid) {
    bool ms = false, as = false;
    int coop = 0;
    if (grid && (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) != cudaSuccess || !coop)) return 0;
    if (!c->cz.ok || !c->cz.csr_built || c->cz.cls.empty() || cluster_smem(c->cz.cls[0], &ms, &as) > CLU_SMEM_MAX) return 0;
    return ms ? 2 : 1;
}

// (the shared-memory limit of a kernel is the process's: always the same value,
// as other threads may be launching it too)
template <int NC, int M, int NW, int LPR, bool MS>
static cudaError_t launch_clu(const CzPlan& z, const CzClass& cl, int grid, size_t smem, cudaStream_t st, CzClu a) {
    if (grid) {
        const bool wide = z.hinst[a.inst_id].rows * LPR > 1024;  // more than two rounds of 512 threads in a product
        const void* k = wide ? (const void*)k_cz_cluster<NC, M, NW, LPR, MS, true, 1024>
                             : (const void*)k_cz_cluster<NC, M, NW, LPR, MS, true, 512>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLU_SMEM_MAX);
        void* args[] = {&a};
        return e == cudaSuccess ? cudaLaunchCooperativeKernel(k, dim3(grid), dim3(wide ? 1024 : 512), args, smem, st) : e;
    }
    // (node blocks whose matrix does not fit on chip take a grid)
    if constexpr (NC == 3 && !MS) {
        return cudaErrorInvalidConfiguration;
    } else {
        auto k = k_cz_cluster<NC, M, NW, LPR, MS, false, 1024>;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLU_SMEM_MAX);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl.ncta * cl.count);
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl.ncta;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, k, &cfg);
        if (e != cudaSuccess) return e;
        if (n < 1) return cudaErrorInvalidConfiguration;
        return cudaLaunchKernelEx(&cfg, k, a);
    }
}

cudaError_t launch_coarse_cluster(isl_ctx* c, bool use_grid, cudaStream_t st, float* work, const float* dinv, double* x64, double tol, double drop,
                                  int max_iter, int big, int cls) {
    CzPlan& z = c->cz;
    bool ms, as;
    const CzClass& cl = big >= 0 ? z.big_cls : z.cls[(size_t)cls];
    const size_t smem = cluster_smem(cl, &ms, &as);
    const int grid = big >= 0 ? z.big_ncta : use_grid ? z.ncta : 0;  // CTAs of the cooperative form
    const size_t na = (size_t)z.nc * z.nrow;
    const bool batch = c->ninst > 1 || c->force_batched;
    CzClu a = {};
    a.lnode = z.lnode.p; a.sofs = z.sofs.p; a.cta = z.cta.p; a.perm = z.perm.p;
    a.dsub = z.dsub.p; a.ainv = z.ainv.p; a.inst = z.inst.p;
    a.order = z.ninst > 1 && big < 0 ? z.order.p + cl.first : nullptr;
    a.cta_stride = z.ncta + 1;
    a.inst_id = big >= 0 ? z.big[big] : 0;
    if (big >= 0) a.cta = z.cta_big.p + (size_t)big * (z.big_ncta + 1);
    a.res = batch ? z.res.p : nullptr;
    a.rp = z.rp.p; a.ci = z.ci.p; a.val = z.cv.p; a.nent = (int)z.nent;
    a.dinv = dinv;
    a.rc = z.rc.p; a.w = work; a.pa = work + na; a.pb = work + 2 * na;
    a.aeq = z.nc == 1 ? nullptr : c->bpad ? c->dbaeq.p : nullptr;
    a.b = c->drhs.p; a.x64 = x64;
    a.rowptr = c->drowptr.p; a.colind = c->dcolind.p; a.val64 = c->dval64.p;
    a.S = c->dscal.p;
    a.tol = tol; a.drop = drop; a.max_iter = max_iter; a.max_gap = coarse_gap(max_iter); a.exact64 = c->have64 ? 1 : 0;
    a.part = reinterpret_cast<float4*>(c->dpart.p); a.bar = c->dbar.p;
    a.inv_smem = as ? 1 : 0;
    if (grid) {
        const cudaError_t e = grid_barrier_start(c, &a.bar_start);
        if (e != cudaSuccess) return e;
    }
    // lanes per row: by the mean row length; in a batch by the element alone, so
    // that an instance's sums do not depend on the others
    const bool wide = batch ? !(c->dim == 2 && c->fedeg == 1) : (double)z.nent > 12.0 * (double)z.nrow;
    if (z.nc == 3) return ms ? launch_clu<3, 6, 8, 8, true>(z, cl, grid, smem, st, a) : launch_clu<3, 6, 8, 8, false>(z, cl, grid, smem, st, a);
    if (z.m == 4) return ms ? launch_clu<1, 4, 8, 8, true>(z, cl, grid, smem, st, a) : launch_clu<1, 4, 8, 8, false>(z, cl, grid, smem, st, a);
    if (wide) return ms ? launch_clu<1, 3, 4, 8, true>(z, cl, grid, smem, st, a) : launch_clu<1, 3, 4, 8, false>(z, cl, grid, smem, st, a);
    return ms ? launch_clu<1, 3, 4, 4, true>(z, cl, grid, smem, st, a) : launch_clu<1, 3, 4, 4, false>(z, cl, grid, smem, st, a);
}

void coarse_args(const isl_ctx* c, CzIter& a) {
    const CzPlan& z = c->cz;
    a.lnode = z.lnode.p;
    a.sofs = z.sofs.p;
    a.dsub = z.dsub.p;
    a.ainv = z.ainv.p;
    a.rc = z.rc.p;
    a.ndp = z.ndp;
}

void launch_coarse(const isl_ctx* c, cudaStream_t st, const CzIter& a, int mode) {
    const CzPlan& z = c->cz;
    CZ_DISPATCH(z, launch_iter, z, st, a, mode);
}

int coarse_spmv_plan(isl_ctx* c) {
    CzPlan& z = c->cz;
    const int g = (int)std::min<int64_t>(z.nslice, (int64_t)SPMV_PER_SM * c->sm_count);
    if (z.bnd_serial == z.serial && z.spmv_ncta == g) return ISL_OK;
    CZ_ALLOC(c, z.bnd, (size_t)g + 1);
    k_cz_bnd<<<g / 256 + 1, 256, 0, c->stream>>>(g, z.nslice, z.soff.p, z.bnd.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 1;
    z.spmv_ncta = g;
    z.bnd_serial = z.serial;
    return ISL_OK;
}
void launch_coarse_spmv(const isl_ctx* c, int kind, cudaStream_t st, const CzSpmv& m) {
    const CzPlan& z = c->cz;
    const bool s16 = z.short_cols && c->use_scol16;
    auto run = [&](auto k16, auto k32) {
        if (s16) launch_chained(k16, z.spmv_ncta, 256, st, m, (const short*)z.col16.p);
        else launch_chained(k32, z.spmv_ncta, 256, st, m, (const int*)z.col.p);
    };
    if (kind == 102) run(k_cz_spmv<4, short>, k_cz_spmv<4, int>);
    else if (kind == 104) run(k_cz_spmv<8, short>, k_cz_spmv<8, int>);
    else run(k_cz_spmv<12, short>, k_cz_spmv<12, int>);
}
void launch_coarse_dir(const isl_ctx* c, cudaStream_t st, int n, const float* z, float* p, const CGScal* S) {
    launch_chained(k_cz_dir, (unsigned)std::min<int64_t>(((int64_t)n + 255) / 256, 16LL * c->sm_count), 256, st, n, z, p, S);
}

}  // namespace isl
