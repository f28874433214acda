// Two-level preconditioner of the mixed CG (single systems).
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
// elasticity 144 -> 19.9 ms (195 iterations instead of 2,257; setup 1.5 ms),
// 20^3 13.6 -> 3.6 ms, 40^3 P2 tetrahedra 38.9 -> 12.4 ms, Q2 160^2 24.2 -> 5.8 ms.
//
// Cost per iteration beyond the one-level solve: the update kernel takes one
// CTA per aggregate and one warp per sub-aggregate, so the restriction and the
// sub-aggregate solve stay inside a warp; one more launch multiplies by the
// dense inverse (its rows for one aggregate per CTA) and prolongs into z.
//
// Determinism: rows of an aggregate are listed in ascending order and summed
// in that order; the coarse entries between aggregates, which several threads
// add to, are summed in 64-bit fixed point.
#include <algorithm>
#include <cmath>
#include <vector>

#include <cub/cub.cuh>

#include "isl_coarse.h"
#include "isl_device.cuh"

namespace isl {

namespace {

constexpr int TB = 64;            // tile of the dense inversion
constexpr int NBIN = 1024;        // bins per axis of the quantile cuts
constexpr int ROW_BITS = 29;      // lnode.w: row, and the constrained components of a padded node block above
constexpr float REG = 1e-5f;      // added to the unit diagonal of the scaled coarse matrices
constexpr int FIX_BITS = 32;      // fixed point of the coarse entries: the largest diagonal entry is 2^32

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
__device__ __forceinline__ void reduce_parts2_df_warp(const float4* part, int n, double& o0, double& o1) {
    o0 = o1 = 0.0;
    if (threadIdx.x >= 32) return;
    df s0 = {0.f, 0.f}, s1 = {0.f, 0.f};
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
    o0 = df_value(warp_sum_df(s0));
    o1 = df_value(warp_sum_df(s1));
}

// ---------------------------------------------------------------------------
// Iteration kernels

// One CTA per aggregate, WPS warps per sub-aggregate.
//   CZ_UPDATE : x += alpha p, r -= alpha q
//   CZ_INIT   : r = b, x = p = 0
//   CZ_RESTART: r = the FP64 residual (reliable update)
// then z = D0^-1 r + P_s D_s^-1 P_s^T r, the aggregate's entries of P^T r, and
// the sums r.r and r.z (without the coarse term, which k_cz_coarse adds).
template <int NC, int M, int NW, int WPS, int MODE>
__global__ void __launch_bounds__(NW * WPS * 32) k_cz_update(CzIter a) {
    constexpr int NT = NW * WPS * 32;
    CGScal* S = a.S;
    if (MODE == CZ_UPDATE && S->done) return;
    if (MODE == CZ_RESTART && !S->rst) return;
    __shared__ double sh[64];
    __shared__ float src[NW * WPS][M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sl = w / WPS, sub = blockIdx.x * NW + sl;
    const int t0 = a.sofs[sub] + (w % WPS) * 32 + lane, t1 = a.sofs[sub + 1];
    const float* __restrict__ p = (a.p2 && !(S->iters & 1)) ? a.p2 : a.p1;
    const float alpha = MODE == CZ_UPDATE ? (float)S->alpha : 0.f;
    float rc[M];
#pragma unroll
    for (int m = 0; m < M; ++m) rc[m] = 0.f;
    float rr = 0.f, rz = 0.f;
    double bb = 0.0;
#pragma unroll 2
    for (int t = t0; t < t1; t += 32 * WPS) {
        const float4 L = __ldg(a.lnode + t);
        const int row = lrow(L);
        const size_t d = (size_t)NC * row;
        float rv[NC], zv[NC], bi[NC * NC];
#pragma unroll
        for (int k = 0; k < NC * NC; ++k) bi[k] = __ldg(a.dinv + (size_t)(NC * NC) * row + k);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (MODE == CZ_UPDATE) {
                a.x[d + c] += alpha * __ldg(p + d + c);
                rv[c] = a.r[d + c] - alpha * __ldg(a.q + d + c);
            } else {
                const int e = a.aeq ? a.aeq[d + c] : (int)(d + c);
                const double v = e >= 0 ? a.b64[e] : 0.0;
                rv[c] = (float)v;
                if (MODE == CZ_INIT) {
                    bb += v * v;
                    a.x[d + c] = 0.f;
                    a.pz[d + c] = 0.f;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            a.r[d + c] = rv[c];
            zv[c] = 0.f;
#pragma unroll
            for (int k = 0; k < NC; ++k) zv[c] += bi[NC * c + k] * rv[k];
            a.z[d + c] = zv[c];
            rr += rv[c] * rv[c];
            rz += rv[c] * zv[c];
        }
        restrict_add<NC, M>(rc, rv, L);
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
    float z1[M];
    const float* __restrict__ D = a.dsub + (size_t)sub * (M * M);
    float rz1 = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
        z1[m] = 0.f;
#pragma unroll
        for (int k = 0; k < M; ++k) z1[m] += __ldg(D + M * m + k) * rc[k];
        rz1 += rc[m] * z1[m];
    }
    if (w % WPS == 0 && lane == 0) rz += rz1;
    for (int t = t0; t < t1; t += 32 * WPS) {  // each thread adds to the entries of z it wrote
        const float4 L = __ldg(a.lnode + t);
        const size_t d = (size_t)NC * lrow(L);
        float o[NC];
        prolong<NC, M>(z1, L, o);
        const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (!((mk >> c) & 1)) a.z[d + c] += o[c];
    }
    if (threadIdx.x < M) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < NW * WPS; ++k) s += src[k][threadIdx.x];
        a.rc[(size_t)blockIdx.x * M + threadIdx.x] = s;
    }
    double trr, trz;
    if (MODE == CZ_INIT) {
        const double b1 = block_sum(bb, sh);
        const double b2 = block_sum((double)rz, sh);
        if (threadIdx.x == 0) { a.part[2 * blockIdx.x] = b1; a.part[2 * blockIdx.x + 1] = b2; }
        if (!last_block(&S->ticket2)) return;
        reduce_parts2(a.part, gridDim.x, sh, trr, trz);
    } else {
        df b1, b2;
        block_sum_df2(rr, rz, reinterpret_cast<float*>(sh), b1, b2);
        if (threadIdx.x == 0) reinterpret_cast<float4*>(a.part)[blockIdx.x] = make_float4(b1.hi, b1.lo, b2.hi, b2.lo);
        if (!last_block(&S->ticket2)) return;
        reduce_parts2_df_warp(reinterpret_cast<const float4*>(a.part), gridDim.x, trr, trz);
    }
    if (threadIdx.x != 0) return;
    S->rr = trr;
    S->rzloc = trz;
    S->ticket2 = 0;
    if (MODE == CZ_UPDATE) {
        S->iters += 1;
        S->absOld = S->absNew;
        if (!(trr == trr) || !(trz == trz)) { S->bad = 1; S->done = 1; }
        else if (trr < S->threshold) S->done = 1;
        else if (trr < S->rrtrig || trr > 1e8 * S->rr_true) S->done = 3;  // dropped enough, or diverging
        else if (S->iters >= S->max_iter) S->done = 2;
    } else if (MODE == CZ_INIT) {
        S->rhsNorm2 = trr;
        S->rr_true = trr;
        S->rr_last = 0.0;
        S->rr_best = trr;
        S->stall = 0;
        S->threshold = a.tol * a.tol * trr;
        S->rrtrig = a.drop * trr;
        S->drop = a.drop;
        S->max_iter = a.max_iter;
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
    if (MODE != CZ_RESTART && S->done) return;
    if (MODE == CZ_RESTART && !S->rst) return;
    __shared__ double sh[64];
    __shared__ float zs[PR][M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n4 = a.ndp / 4;
    const float4* __restrict__ rc4 = reinterpret_cast<const float4*>(a.rc);
    for (int j = w; j < M * PR; j += TW) {
        const int m = j % M;
        const float4* __restrict__ row = reinterpret_cast<const float4*>(a.ainv + (size_t)(blockIdx.x * M + m) * a.ndp);
        float s = 0.f;
#pragma unroll 4
        for (int k = (j / M) * 32 + lane; k < n4; k += 32 * PR) {
            const float4 v = __ldg(row + k), u = __ldg(rc4 + k);
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
        rz += zc[m] * __ldg(a.rc + (size_t)blockIdx.x * M + m);
    }
    const int t1 = a.sofs[(blockIdx.x + 1) * NW];
    for (int t = a.sofs[blockIdx.x * NW] + (int)threadIdx.x; t < t1; t += TW * 32) {
        const float4 L = __ldg(a.lnode + t);
        const size_t d = (size_t)NC * lrow(L);
        float o[NC];
        prolong<NC, M>(zc, L, o);
        const int mk = NC == 3 ? lmask(L) : 0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
            if (!((mk >> c) & 1)) a.z[d + c] += o[c];
    }
    if (threadIdx.x == 0) reinterpret_cast<float2*>(a.part)[blockIdx.x] = make_float2(rz, 0.f);
    if (!last_block(&S->ticket2)) return;
    const double tot = reduce_parts_df(reinterpret_cast<const float2*>(a.part), gridDim.x);
    if (threadIdx.x != 0) return;
    S->ticket2 = 0;
    const double rzn = S->rzloc + tot;
    S->absNew = rzn;
    if (MODE == CZ_UPDATE) S->beta = rzn / S->absOld;
    else if (MODE == CZ_INIT) { S->absOld = rzn; S->beta = 0.0; }
    else {
        S->beta = S->fresh ? 0.0 : rzn / S->absOld;
        S->done = 0;
        S->rst = 0;
    }
    // not positive: the matrix or the inverse is not definite; the host solves one-level
    if (!(rzn > 0.0)) { S->bad = 1; S->done = 1; }
}

// p = z + beta p (where the product does not fold the direction update)
__global__ void __launch_bounds__(256) k_cz_dir(int n, const float* __restrict__ z, float* __restrict__ p, const CGScal* S) {
    if (S->done) return;
    const float beta = (float)S->beta;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) p[i] = fmaf(beta, p[i], z[i]);
}

// ---------------------------------------------------------------------------
// Numeric setup, once per assembly

// largest diagonal entry (its bits order as integers)
template <typename T>
__global__ void k_cz_amax(int n, const int* __restrict__ diag, const T* __restrict__ val, int* __restrict__ out) {
    float m = 0.f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = fabsf((float)val[diag[i]]);
        if (v < INFINITY) m = fmaxf(m, v);
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_int(m));
}

__device__ inline float fix_scale(int amax_bits) {  // 2^(FIX_BITS - e), amax < 2^e
    const int e = ((amax_bits >> 23) & 255) - 126;
    return ldexpf(1.f, FIX_BITS - e);
}

// Galerkin blocks: CTA per aggregate, warp per sub-aggregate, lane per row.
// The entries inside a sub-aggregate and inside the aggregate are summed in
// registers and by fixed shuffle trees; those towards a later aggregate go to
// acc in fixed point, one run of equal aggregates of a row at a time (the
// entries towards earlier ones follow by symmetry).
template <int NC, int M, int NW>
__global__ void __launch_bounds__(NW * 32) k_cz_galerkin(CzMat A, const float4* __restrict__ lnode, const float4* __restrict__ yrow,
                                                         const int* __restrict__ sofs, int ndp, const int* __restrict__ amax,
                                                         unsigned long long* __restrict__ acc, float* __restrict__ dsub,
                                                         float* __restrict__ dagg) {
    __shared__ float own[NW][M * M];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x, sub = I * NW + w;
    const float scale = fix_scale(*amax);
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
            outer(Tc, L, o, false);
            unsigned long long* dst = acc + (size_t)(I * M) * ndp + (size_t)J * M;
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
        if (NC == 3) {
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

// the scaled coarse matrix, padded with the identity to whole tiles
template <int M>
__global__ void k_cz_form(int nd, int ndp, const unsigned long long* __restrict__ acc, const float* __restrict__ dagg,
                          const float* __restrict__ s, const int* __restrict__ amax, float* __restrict__ A) {
    const float inv = 1.f / fix_scale(*amax);
    const int j = blockIdx.x * 32 + (threadIdx.x & 31);
    for (int i = blockIdx.y * 32 + (threadIdx.x >> 5); i < blockIdx.y * 32 + 32; i += 8) {
        float v = 0.f;
        if (i == j) v = 1.f + REG;
        else if (i < nd && j < nd) {
            const int I = i / M, J = j / M;
            if (I == J) v = 0.5f * (dagg[(size_t)I * M * M + (i % M) * M + j % M] + dagg[(size_t)I * M * M + (j % M) * M + i % M]);
            else v = (float)(long long)acc[I < J ? (size_t)i * ndp + j : (size_t)j * ndp + i] * inv;
            v *= s[i] * s[j];
        }
        A[(size_t)i * ndp + j] = v;
    }
}

// Dense inversion of the coarse matrix (symmetric positive definite, unit
// diagonal) by block sweeps without pivoting, TB rows per step.  Sweeping
// block k takes A_kk to -D^-1, A_Ik to A_Ik D^-1 and A_IJ to A_IJ - A_Ik D^-1
// A_kJ, keeps the matrix symmetric, and leaves -A^-1 after the last block; only
// the tiles on and below the diagonal are stored and updated.
//
// Two launches per step: the panel kernel forms G_I = A_Ik D^-1 for every tile
// row I and saves the old panel P_I = A_Ik; the update kernel subtracts
// G_I P_J^T from the other tiles.  The inverse of the next diagonal tile is
// computed by the CTA that updates it, beside the other tiles' updates: a warp
// inverts 32 x 32 in registers (a lane per row), and the tile is two of those
// around a Schur complement.  1.5 ms of setup at 64^3 (1,764 rows) with the
// Galerkin blocks; pivoting a whole tile with one block barrier per row took
// 78 us a step, 3.3 ms in all.

// inverse of the 32 x 32 matrix in X (leading dimension TB + 1) by one warp
__device__ __forceinline__ void warp_inv32(float* X) {
    const int l = threadIdx.x & 31;
    float a[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) a[c] = X[l * (TB + 1) + c];
#pragma unroll
    for (int p = 0; p < 32; ++p) {
        const float ip = 1.f / fmaxf(__shfl_sync(0xffffffffu, a[p], p), 0.1f * REG);
        const float f = l == p ? 1.f - ip : a[p] * ip;  // row l minus f times the pivot row; the pivot row scales by ip
#pragma unroll
        for (int c = 0; c < 32; ++c)
            if (c != p) a[c] -= f * __shfl_sync(0xffffffffu, a[c], p);
        a[p] = l == p ? ip : -f;
    }
#pragma unroll
    for (int c = 0; c < 32; ++c) X[l * (TB + 1) + c] = a[c];
    __syncwarp();
}

// inverse of the symmetric TB x TB matrix D in shared memory by 256 threads;
// T: scratch of the same size
__device__ __forceinline__ void tile_inv(float (*D)[TB + 1], float (*T)[TB + 1]) {
    const int r = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 4;  // 32 rows, 4 columns per thread
    if (threadIdx.x < 32) warp_inv32(&D[0][0]);                  // A <- A^-1
    __syncthreads();
    {   // T_01 = A^-1 B
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int m = 0; m < 32; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] += D[r][m] * D[m][32 + c0 + c];
#pragma unroll
        for (int c = 0; c < 4; ++c) T[r][32 + c0 + c] = o[c];
    }
    __syncthreads();
    {   // C <- C - B^T A^-1 B
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int m = 0; m < 32; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] += D[m][32 + r] * T[m][32 + c0 + c];
#pragma unroll
        for (int c = 0; c < 4; ++c) D[32 + r][32 + c0 + c] -= o[c];
    }
    __syncthreads();
    if (threadIdx.x < 32) warp_inv32(&D[32][32]);  // C <- S^-1
    __syncthreads();
    {   // T_10^T = A^-1 B S^-1
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int m = 0; m < 32; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] += T[r][32 + m] * D[32 + m][32 + c0 + c];
#pragma unroll
        for (int c = 0; c < 4; ++c) { D[r][32 + c0 + c] = -o[c]; D[32 + c0 + c][r] = -o[c]; }
    }
    __syncthreads();
    {   // A^-1 + (A^-1 B) S^-1 (A^-1 B)^T
        float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int m = 0; m < 32; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] -= D[r][32 + m] * T[c0 + c][32 + m];
#pragma unroll
        for (int c = 0; c < 4; ++c) D[r][c0 + c] += o[c];
    }
    __syncthreads();
}

// the inverse of the first diagonal tile
__global__ void __launch_bounds__(256) k_gj_first(const float* __restrict__ A, int n, float* __restrict__ Dinv) {
    __shared__ float D[TB][TB + 1], T[TB][TB + 1];
    for (int e = threadIdx.x; e < TB * TB; e += 256) D[e / TB][e % TB] = A[(size_t)(e / TB) * n + e % TB];
    __syncthreads();
    tile_inv(D, T);
    for (int e = threadIdx.x; e < TB * TB; e += 256) Dinv[e] = D[e / TB][e % TB];
}

// C[4 ty + r][tx + 16 c] += sum_m X[4 ty + r][m] Y[tx + 16 c][m]
__device__ __forceinline__ void tile_mul(const float (*X)[TB + 1], const float (*Y)[TB + 1], float (&o)[4][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
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

// G_I = A_Ik D^-1, P_I = A_Ik (A_Ik = A_kI^T above the diagonal)
__global__ void __launch_bounds__(256) k_gj_panel(const float* __restrict__ A, int n, int k, const float* __restrict__ Dinv,
                                                  float* __restrict__ G, float* __restrict__ P) {
    __shared__ float X[TB][TB + 1], D[TB][TB + 1];
    const int I = blockIdx.x, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (I == k) return;
    for (int e = threadIdx.x; e < TB * TB; e += 256) {
        const int r = e / TB, c = e % TB;
        if (I > k) X[r][c] = A[(size_t)(I * TB + r) * n + k * TB + c];
        else X[c][r] = A[(size_t)(k * TB + r) * n + I * TB + c];
        D[r][c] = Dinv[e];
    }
    __syncthreads();
    float o[4][4] = {};
    tile_mul(X, D, o);  // D^-1 is symmetric
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) G[(size_t)(I * TB + 4 * ty + r) * TB + tx + 16 * c] = o[r][c];
    for (int e = threadIdx.x; e < TB * TB; e += 256) P[(size_t)I * TB * TB + e] = X[e / TB][e % TB];
}

__global__ void __launch_bounds__(256) k_gj_update(float* __restrict__ A, int n, int k, float* __restrict__ Dinv,
                                                   float* __restrict__ Dnext, const float* __restrict__ G,
                                                   const float* __restrict__ P) {
    __shared__ float X[TB][TB + 1], Y[TB][TB + 1];
    // tile (I, J), J <= I, of the linear index; the next diagonal tile comes first
    int t = blockIdx.x;
    const int nt = n / TB, first = k + 1 < nt ? (k + 1) * (k + 2) / 2 + k + 1 : -1;
    if (first >= 0) t = t == 0 ? first : (t <= first ? t - 1 : t);
    int I = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    while (I * (I + 1) / 2 > t) --I;
    const int J = t - I * (I + 1) / 2, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float* g = A + (size_t)(I * TB) * n + J * TB;
    if (I == k || J == k) {
        for (int e = threadIdx.x; e < TB * TB; e += 256) {
            const int r = e / TB, c = e % TB;
            if (I == J) g[(size_t)r * n + c] = -Dinv[e];
            else if (J == k) g[(size_t)r * n + c] = G[(size_t)(I * TB + r) * TB + c];
            else g[(size_t)r * n + c] = G[(size_t)(J * TB + c) * TB + r];
        }
        return;
    }
    for (int e = threadIdx.x; e < TB * TB; e += 256) {
        X[e / TB][e % TB] = G[(size_t)I * TB * TB + e];
        Y[e / TB][e % TB] = P[(size_t)J * TB * TB + e];
    }
    float a[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) a[r][c] = g[(size_t)(4 * ty + r) * n + tx + 16 * c];
    __syncthreads();
    float o[4][4] = {};
    tile_mul(X, Y, o);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            a[r][c] -= o[r][c];
            g[(size_t)(4 * ty + r) * n + tx + 16 * c] = a[r][c];
        }
    if (I != J || I != k + 1) return;
    __syncthreads();  // the next diagonal tile: its inverse
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) X[4 * ty + r][tx + 16 * c] = a[r][c];
    __syncthreads();
    tile_inv(X, Y);
    for (int e = threadIdx.x; e < TB * TB; e += 256) Dnext[e] = X[e / TB][e % TB];
}

// undo the sign and the scaling, and fill the upper triangle from the lower
__global__ void k_cz_unscale(int nd, int ndp, const float* __restrict__ A, const float* __restrict__ s, float* __restrict__ out) {
    __shared__ float T[32][33];
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
                            const int32_t* __restrict__ edof, const double* __restrict__ X, int D, float* __restrict__ P) {
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
            P[o * D + d] = (float)v;
        }
    }
}

__global__ void k_cz_eqrow(int n3, const int* __restrict__ aeq, int* __restrict__ eqrow) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n3 && aeq[t] >= 0) eqrow[aeq[t]] = t / 3;
}

// point (w: the component, NC = 1, or the mask of constrained components) of every row
template <int NC>
__global__ void k_cz_rowpts(int64_t ndo, int ncomp, const int32_t* __restrict__ eq, const int* __restrict__ eqrow, int D,
                            const float* __restrict__ P, float4* __restrict__ xr) {
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= ndo) return;
    float4 v = make_float4(P[o * D], P[o * D + 1], D == 3 ? P[o * D + 2] : 0.f, 0.f);
    if (NC == 1) {
        for (int c = 0; c < ncomp; ++c) {
            const int e = eq[o * ncomp + c];
            v.w = __int_as_float(c);
            if (e >= 0) xr[e] = v;
        }
    } else {
        int first = -1, mask = 0;
        for (int c = 0; c < 3; ++c) {
            const int e = eq[o * 3 + c];
            if (e < 0) mask |= 1 << c;
            else if (first < 0) first = e;
        }
        if (first < 0) return;
        v.w = __int_as_float(mask);
        xr[eqrow ? eqrow[first] : first / 3] = v;
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

__global__ void k_cz_bounds(int n, const float4* __restrict__ xr, unsigned* __restrict__ mm) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v[3] = {xr[i].x, xr[i].y, xr[i].z};
#pragma unroll
        for (int d = 0; d < 3; ++d) { lo[d] = fminf(lo[d], v[d]); hi[d] = fmaxf(hi[d], v[d]); }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
        if ((threadIdx.x & 31) == 0) { atomicMin(mm + d, f_order(lo[d])); atomicMax(mm + 3 + d, f_order(hi[d])); }
    }
}

struct Box3 { float lo[3], inv[3]; int m[3]; };  // m: boxes per direction

__device__ inline int bin_of(const Box3& b, int d, float x) {
    return min(NBIN - 1, max(0, (int)((x - b.lo[d]) * b.inv[d])));
}

__global__ void k_cz_hist(int n, Box3 b, const float4* __restrict__ xr, int* __restrict__ hist) {
    __shared__ int h[3 * NBIN];
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

// raw key of every row: (box, component) and sub-box; cut[d][bin] is the
// half-box index along d
template <int NC, int NW>
__global__ void k_cz_key(int n, Box3 b, const unsigned short* __restrict__ cut, int ncomp, const float4* __restrict__ xr,
                         int* __restrict__ key, int* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = xr[i];
        const int h0 = cut[bin_of(b, 0, v.x)], h1 = cut[NBIN + bin_of(b, 1, v.y)], h2 = cut[2 * NBIN + bin_of(b, 2, v.z)];
        int g = ((h2 >> 1) * b.m[1] + (h1 >> 1)) * b.m[0] + (h0 >> 1);
        if (NC == 1) g = g * ncomp + __float_as_int(v.w);
        const int s = (h0 & 1) | (h1 & 1) << 1 | (NW == 8 ? (h2 & 1) << 2 : 0);
        key[i] = g * NW + s;
        atomicAdd(&cnt[g * NW + s], 1);
    }
}

template <int NW>
__global__ void k_cz_rekey(int n, const int* __restrict__ map, int* __restrict__ key, int* __restrict__ row) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = key[i];
        key[i] = map[k / NW] * NW + k % NW;
        row[i] = i;
    }
}

// centre and rms radius of every aggregate, then the rows' scaled positions
template <int NC, int NW>
__global__ void __launch_bounds__(NW * 32) k_cz_nodes(const int* __restrict__ sofs, const int* __restrict__ list,
                                                      const int* __restrict__ key, const float4* __restrict__ xr,
                                                      float4* __restrict__ lnode, float4* __restrict__ yrow) {
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
        y.w = __int_as_float(row | (NC == 3 ? __float_as_int(v.w) << ROW_BITS : 0));
        lnode[t] = y;
        y.w = __int_as_float(key[t]);
        yrow[row] = y;
    }
}

// Number of aggregates for n rows: about 60 rows each, at most 150 (300 for
// the largest systems).  More aggregates take fewer iterations; the dense
// inversion grows with their cube.  Measured with setup (node blocks): 2,366
// rows 3.33 ms with 24 aggregates, 2.98 with 50, 3.10 with 100; 31,744 rows
// 5.50 with 150, 5.70 with 300; 270,400 rows 21.9 with 150, 20.0 with 300,
// 21.3 with 400.
int target_aggs(int64_t n) {
    return (int)std::clamp<int64_t>(n / 60, 8, std::clamp<int64_t>(n / 900, 150, 300));
}

unsigned grid_for(const isl_ctx* c, int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8LL * c->sm_count)); }

template <int NC, int M, int NW>
int build_plan(isl_ctx* c, CzPlan& z) {
    cudaStream_t st = c->stream;
    const int D = c->dim, n = (int)z.nrow;
    DBuf<float> P;
    DBuf<float4> xr;
    DBuf<int32_t> eqrow, hist, key, key2, row, list, cnt, map;
    DBuf<unsigned> mm;
    DBuf<unsigned short> dcut;
    DBuf<char> tmp;
    ISL_CHECK_CUDA(c, P.alloc((size_t)c->ndofobj * D));
    ISL_CHECK_CUDA(c, xr.alloc(n));
    ISL_CHECK_CUDA(c, mm.alloc(6));
    ISL_CHECK_CUDA(c, hist.alloc(3 * NBIN));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(mm.p, 0xff, 3 * 4, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(mm.p + 3, 0, 3 * 4, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(hist.p, 0, 3 * NBIN * 4, st));
    k_cz_points<<<(unsigned)((c->nelem + 255) / 256), 256, 0, st>>>(c->shape, c->ngeom, c->nfun, c->nelem, c->dconn.p,
                                                                     c->dedof.p, c->dX.p, D, P.p);
    if (NC == 3 && c->bpad) {
        ISL_CHECK_CUDA(c, eqrow.alloc((size_t)c->neq));
        k_cz_eqrow<<<(3 * n + 255) / 256, 256, 0, st>>>(3 * n, c->dbaeq.p, eqrow.p);
        c->launches += 1;
    }
    k_cz_rowpts<NC><<<(unsigned)((c->ndofobj + 255) / 256), 256, 0, st>>>(c->ndofobj, c->ncomp, c->deq.p, eqrow.p, D, P.p, xr.p);
    const unsigned g = grid_for(c, n);
    k_cz_bounds<<<g, 256, 0, st>>>(n, xr.p, mm.p);
    unsigned hmm[6];
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hmm, mm.p, sizeof(hmm), cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    Box3 b;
    double L[3] = {0, 0, 0}, Lmax = 0;
    for (int d = 0; d < 3; ++d) {
        const float lo = f_unorder(hmm[d]), hi = f_unorder(hmm[3 + d]);
        L[d] = d < D ? (double)hi - lo : 0.0;
        if (!(L[d] >= 0.0) || !std::isfinite(L[d])) return ISL_OK;  // no usable coordinates: one-level
        Lmax = std::max(Lmax, L[d]);
        b.lo[d] = lo;
        b.inv[d] = L[d] > 0.0 ? (float)(NBIN / L[d]) : 0.f;
    }
    if (!(Lmax > 0.0)) return ISL_OK;
    k_cz_hist<<<std::min(g, (unsigned)c->sm_count), 256, 0, st>>>(n, b, xr.p, hist.p);
    std::vector<int32_t> hh(3 * NBIN);
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hh.data(), hist.p, hh.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    // near-cubic boxes: the edge h that gives the target number of them
    const int comps = NC == 1 ? c->ncomp : 1;
    const int target = std::max(1, target_aggs(z.nrow) / comps);
    double vol = 1.0;
    int nd = 0;
    for (int d = 0; d < D; ++d)
        if (L[d] > 1e-3 * Lmax) { vol *= L[d]; ++nd; }
    double h = std::pow(vol / target, 1.0 / nd);
    for (;;) {
        int64_t tot = 1;
        for (int d = 0; d < 3; ++d) {
            b.m[d] = d < D ? std::max(1, (int)std::lround(L[d] / h)) : 1;
            tot *= b.m[d];
        }
        if (tot <= std::max(target, 1)) break;
        h *= 1.02;
    }
    const int nbox = b.m[0] * b.m[1] * b.m[2] * comps;
    // cuts at the quantiles of the rows, two half-boxes per box
    std::vector<unsigned short> cut(3 * NBIN, 0);
    for (int d = 0; d < D; ++d) {
        const int64_t parts = 2 * b.m[d];
        int64_t run = 0;
        for (int k = 0; k < NBIN; ++k) {
            const int64_t mid = run + hh[d * NBIN + k] / 2;
            cut[d * NBIN + k] = (unsigned short)std::min<int64_t>(parts - 1, mid * parts / std::max(n, 1));
            run += hh[d * NBIN + k];
        }
    }
    ISL_CHECK_CUDA(c, dcut.alloc(3 * NBIN));
    ISL_CHECK_CUDA(c, key.alloc(n));
    ISL_CHECK_CUDA(c, key2.alloc(n));
    ISL_CHECK_CUDA(c, row.alloc(n));
    ISL_CHECK_CUDA(c, list.alloc(n));
    ISL_CHECK_CUDA(c, cnt.alloc((size_t)nbox * NW));
    ISL_CHECK_CUDA(c, map.alloc(nbox));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(dcut.p, cut.data(), cut.size() * 2, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(cnt.p, 0, (size_t)nbox * NW * 4, st));
    k_cz_key<NC, NW><<<g, 256, 0, st>>>(n, b, dcut.p, c->ncomp, xr.p, key.p, cnt.p);
    std::vector<int32_t> hc((size_t)nbox * NW), hmap(nbox, -1), so;
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(hc.data(), cnt.p, hc.size() * 4, cudaMemcpyDeviceToHost, st));
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
    int32_t run = 0, na = 0;
    for (int k = 0; k < nbox; ++k) {
        int32_t tot = 0;
        for (int s = 0; s < NW; ++s) tot += hc[(size_t)k * NW + s];
        if (!tot) continue;
        hmap[k] = na++;
        for (int s = 0; s < NW; ++s) { so.push_back(run); run += hc[(size_t)k * NW + s]; }
    }
    so.push_back(run);
    z.nagg = na;
    z.nd = na * M;
    z.ndp = (z.nd + TB - 1) / TB * TB;
    ISL_CHECK_CUDA(c, z.sofs.alloc(so.size()));
    ISL_CHECK_CUDA(c, z.lnode.alloc(n));
    ISL_CHECK_CUDA(c, z.yrow.alloc(n));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(z.sofs.p, so.data(), so.size() * 4, cudaMemcpyHostToDevice, st));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(map.p, hmap.data(), hmap.size() * 4, cudaMemcpyHostToDevice, st));
    k_cz_rekey<NW><<<g, 256, 0, st>>>(n, map.p, key.p, row.p);
    int bits = 1;
    while ((1 << bits) < na * NW) ++bits;
    size_t tb = 0;
    ISL_CHECK_CUDA(c, cub::DeviceRadixSort::SortPairs(nullptr, tb, key.p, key2.p, row.p, list.p, n, 0, bits, st));
    ISL_CHECK_CUDA(c, tmp.alloc(std::max<size_t>(tb, 1)));
    ISL_CHECK_CUDA(c, cub::DeviceRadixSort::SortPairs(tmp.p, tb, key.p, key2.p, row.p, list.p, n, 0, bits, st));
    k_cz_nodes<NC, NW><<<na, NW * 32, 0, st>>>(z.sofs.p, list.p, key2.p, xr.p, z.lnode.p, z.yrow.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    ISL_CHECK_CUDA(c, z.dsub.alloc((size_t)na * NW * M * M));
    ISL_CHECK_CUDA(c, z.dagg.alloc((size_t)na * M * M));
    ISL_CHECK_CUDA(c, z.scale.alloc(z.ndp));
    ISL_CHECK_CUDA(c, z.rc.alloc(z.ndp));
    ISL_CHECK_CUDA(c, z.acc.alloc((size_t)z.ndp * z.ndp));
    ISL_CHECK_CUDA(c, z.a.alloc((size_t)z.ndp * z.ndp));
    ISL_CHECK_CUDA(c, z.ainv.alloc((size_t)z.ndp * z.ndp));
    ISL_CHECK_CUDA(c, z.panel.alloc((size_t)2 * TB * z.ndp + 2 * TB * TB));
    ISL_CHECK_CUDA(c, z.amax.alloc(1));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.rc.p, 0, (size_t)z.ndp * 4, st));  // the padding stays zero
    ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));  // the scratch buffers above go out of scope
    c->launches += 10;
    z.ok = true;
    return ISL_OK;
}

template <int NC, int M, int NW>
int numeric(isl_ctx* c, CzPlan& z, const CzMat& A) {
    cudaStream_t st = c->stream;
    const int ndp = z.ndp, nt = ndp / TB;
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.acc.p, 0, (size_t)ndp * ndp * 8, st));
    ISL_CHECK_CUDA(c, cudaMemsetAsync(z.amax.p, 0, 4, st));
    const unsigned g = grid_for(c, c->neq);
    if (c->have64) k_cz_amax<double><<<g, 256, 0, st>>>((int)c->neq, c->ddiag.p, c->dval64.p, z.amax.p);
    else k_cz_amax<float><<<g, 256, 0, st>>>((int)c->neq, c->ddiag.p, c->dval32.p, z.amax.p);
    k_cz_galerkin<NC, M, NW><<<z.nagg, NW * 32, 0, st>>>(A, z.lnode.p, z.yrow.p, z.sofs.p, ndp, z.amax.p, z.acc.p, z.dsub.p,
                                                         z.dagg.p);
    k_cz_sub_inv<M><<<(z.nagg * NW + 63) / 64, 64, 0, st>>>(z.nagg * NW, z.dsub.p);
    k_cz_scale<M><<<(z.nagg + 127) / 128, 128, 0, st>>>(z.nagg, z.dagg.p, z.scale.p);
    const dim3 g32(ndp / 32, ndp / 32);
    k_cz_form<M><<<g32, 256, 0, st>>>(z.nd, ndp, z.acc.p, z.dagg.p, z.scale.p, z.amax.p, z.a.p);
    float *G = z.panel.p, *P = G + (size_t)TB * ndp, *D[2] = {P + (size_t)TB * ndp, P + (size_t)TB * ndp + TB * TB};
    k_gj_first<<<1, 256, 0, st>>>(z.a.p, ndp, D[0]);
    for (int k = 0; k < nt; ++k) {
        if (nt > 1) k_gj_panel<<<nt, 256, 0, st>>>(z.a.p, ndp, k, D[k & 1], G, P);
        k_gj_update<<<nt * (nt + 1) / 2, 256, 0, st>>>(z.a.p, ndp, k, D[k & 1], D[(k + 1) & 1], G, P);
    }
    k_cz_unscale<<<g32, 256, 0, st>>>(z.nd, ndp, z.a.p, z.scale.p, z.ainv.p);
    ISL_CHECK_CUDA(c, cudaGetLastError());
    c->launches += 7 + 2 * nt;
    return ISL_OK;
}

template <int NC, int M, int NW, int WPS>
void launch_iter_w(const CzPlan& z, cudaStream_t st, const CzIter& a, int mode) {
    const unsigned g = (unsigned)z.nagg, t = NW * WPS * 32;
    if (mode == CZ_UPDATE) {
        k_cz_update<NC, M, NW, WPS, CZ_UPDATE><<<g, t, 0, st>>>(a);
        k_cz_coarse<NC, M, NW, WPS, CZ_UPDATE><<<g, t, 0, st>>>(a);
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

int coarse_plan(isl_ctx* c, int nc, int64_t nrow) {
    CzPlan& z = c->cz;
    if (z.serial == c->pattern_serial && z.nc == nc) return ISL_OK;
    z.ok = false;
    z.num_serial = -1;
    z.nc = nc;
    z.m = nc == 3 ? 6 : 1 + c->dim;
    z.nrow = nrow;
    z.serial = c->pattern_serial;
    if (nrow >= (1 << ROW_BITS) || c->fedeg > 2 || (c->fedeg == 2 && c->shape == ISL_HEX) || c->ninst != 1) return ISL_OK;
    return CZ_DISPATCH(z, build_plan, c, z);
}

int coarse_numeric(isl_ctx* c, const CzMat& A) {
    CzPlan& z = c->cz;
    if (z.num_serial == c->asm_serial) return ISL_OK;
    const int rc = CZ_DISPATCH(z, numeric, c, z, A);
    if (rc == ISL_OK) z.num_serial = c->asm_serial;
    return rc;
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

void launch_coarse_dir(const isl_ctx* c, cudaStream_t st, int n, const float* z, float* p, const CGScal* S) {
    k_cz_dir<<<(unsigned)std::min<int64_t>(((int64_t)n + 255) / 256, 16LL * c->sm_count), 256, 0, st>>>(n, z, p, S);
}

}  // namespace isl
