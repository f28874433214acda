// FP64 solves of small systems in one cooperative launch: the Jacobi CG of
// solve_fp64 and the BiCGSTAB of isl_krylov.cu, the same recurrences with FP64
// vectors, matrix and sums.
//
// The graph paths launch three (five) kernels per iteration, each with a
// reduction tail: 22-25 us (43 us) whatever the size.  Here one CTA per SM owns
// a range of rows, balanced by stored entries, with its rows of the matrix and
// its vectors in shared memory.  The columns a CTA touches are renumbered (a
// bitmap and its prefix counts), and the CTA keeps the direction at all of
// them, own rows and halo, updating the halo itself from the vectors their
// owners publish.  So the product reads shared memory only, a direction update
// needs no barrier of its own, and an iteration has one grid barrier per
// reduction: two for CG, three for BiCGSTAB.  us per iteration: Q2 121 x 77
// (582k entries) 22.4 -> 10.6, 24,840-equation elasticity (1.8M) 25.0 -> 12.4,
// heat::Static Q2 61 x 47 42.8 -> 13.9.  What is left is FP64: about 1.2 FMAs per
// clock and SM (5 us of products at 1.8M entries), some 90 cycles of latency
// per dependent add in the sums (1.4 us each), a division per scalar, and the
// barriers (1-2 us each).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <vector>

#include "isl_device.cuh"
#include "isl_internal.h"

namespace isl {

namespace {

// threads per CTA: CG 10.7 us an iteration with 1024, 11.4 with 512 (Q2 121 x 77);
// BiCGSTAB 13.7 with 512, 14.2 with 1024 (heat Q2 61 x 47)
constexpr int OT_CG = 1024, OT_BI = 512;
constexpr size_t OL_SMEM_MAX = 224 * 1024;
// CG beside other such solves of this process: half the threads and at most half the
// shared memory, so that the grids of two solves are resident at once.  The sums
// and products of a row do not depend on the threads: the same bits.  Eight host
// threads, Q2 90 x 90 (32k rows): 241 solves a second, 150 with one grid at a time, 186
// as graphs of kernels; Q1 100 x 100: 876, 453 and 558.
constexpr int OT_CG_HALF = 512;
constexpr size_t OL_SMEM_HALF = 112 * 1024;

struct OlArgs {
    int n;
    const int *rp, *ci, *diag, *row0;  // row0: first row of every CTA
    const double *val, *b;
    int R, E, H, vals_in, lanes;       // capacities: rows, entries, columns; values in shared memory; lanes per row
    double *g1, *g2, *g3;              // published vectors
    double *x;
    double* part;                      // [4 slots][2][CTAs]
    unsigned* bar;
    unsigned bar_start;                // count at which the grid barrier starts
    OlScal* S;
    double tol;
    int max_iter;
};

// shared-memory layout: nd vectors over the rows, nh over the columns.  share: the
// bitmap and its counts, needed while the columns are numbered only, take the room
// of the row vectors (the layout of whole-SM launches keeps them apart: 0.7 %
// faster, as the vectors' banks fall)
struct OlMem {
    double *row, *hal, *vals;
    int *rps, *hc, *li;
    unsigned *bits;
    int* pre;
    unsigned short* cols;
};
__host__ __device__ inline size_t ol_row_words(int n, int R, int nd, bool share) {
    const size_t W = (n + 31) / 32, v = (size_t)nd * R;  // a bitmap word and a count: 8 bytes
    return share && W > v ? W : v;
}
__host__ __device__ inline size_t ol_bytes(int n, int R, int E, int H, int nd, int nh, bool vals, bool share) {
    const size_t W = (n + 31) / 32;
    return 8 * (ol_row_words(n, R, nd, share) + (size_t)nh * H + (vals ? (size_t)E : 0)) +
           4 * ((size_t)R + 1 + H + R + (share ? 0 : 2 * W)) + 2 * (size_t)E + 16;
}
template <bool SHARE>
__device__ inline OlMem ol_mem(const OlArgs& a, unsigned char* p, int nd, int nh) {
    OlMem m;
    const int W = (a.n + 31) / 32;
    m.row = reinterpret_cast<double*>(p);
    m.hal = m.row + ol_row_words(a.n, a.R, nd, SHARE);
    m.vals = m.hal + (size_t)nh * a.H;
    m.rps = reinterpret_cast<int*>(m.vals + (a.vals_in ? a.E : 0));
    m.hc = m.rps + a.R + 1;
    m.li = m.hc + a.H;
    m.bits = SHARE ? reinterpret_cast<unsigned*>(m.row) : reinterpret_cast<unsigned*>(m.li + a.R);
    m.pre = reinterpret_cast<int*>(m.bits + W);
    m.cols = SHARE ? reinterpret_cast<unsigned short*>(m.li + a.R) : reinterpret_cast<unsigned short*>(m.pre + W);
    return m;
}

// the CTA's matrix rows and its column numbering; returns the number of columns
template <int OT>
__device__ inline int ol_setup(const OlArgs& a, const OlMem& m, int r0, int nr, int e0, int ne) {
    __shared__ int wsum[OT / 32];
    __shared__ int total;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int W = (a.n + 31) / 32;
    for (int k = tid; k < W; k += OT) m.bits[k] = 0u;
    for (int i = tid; i <= nr; i += OT) m.rps[i] = a.rp[r0 + i] - e0;
    __syncthreads();
    for (int k = tid; k < ne; k += OT) {
        const int j = a.ci[e0 + k];
        atomicOr(&m.bits[j >> 5], 1u << (j & 31));
        if (a.vals_in) m.vals[k] = a.val[e0 + k];
    }
    for (int i = tid; i < nr; i += OT) atomicOr(&m.bits[(r0 + i) >> 5], 1u << ((r0 + i) & 31));
    __syncthreads();
    // exclusive prefix counts of the words, a run of words per thread
    const int per = (W + OT - 1) / OT, k0 = min(W, tid * per), k1 = min(W, k0 + per);
    int cnt = 0;
    for (int k = k0; k < k1; ++k) cnt += __popc(m.bits[k]);
    int inc = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (tid == 0) {
        int s = 0;
        for (int k = 0; k < OT / 32; ++k) { const int t = wsum[k]; wsum[k] = s; s += t; }
        total = s;
    }
    __syncthreads();
    const int nh = total;
    if (nh > a.H) return nh;
    int pos = wsum[w] + inc - cnt;
    for (int k = k0; k < k1; ++k) {
        m.pre[k] = pos;
        for (unsigned b = m.bits[k]; b; b &= b - 1) m.hc[pos++] = 32 * k + __ffs(b) - 1;
    }
    __syncthreads();
    auto local = [&](int j) { return m.pre[j >> 5] + __popc(m.bits[j >> 5] & ((1u << (j & 31)) - 1u)); };
    for (int k = tid; k < ne; k += OT) m.cols[k] = (unsigned short)local(a.ci[e0 + k]);
    for (int i = tid; i < nr; i += OT) m.li[i] = local(r0 + i);
    __syncthreads();
    return nh;
}

// out_i = sum over row i of A times the column vector v; f(i, out_i) runs in one
// lane per row.  L lanes per row: a warp's FP64 instruction occupies the pipe
// for 16 cycles whatever its lanes hold, so short rows take few lanes (the
// shuffle tree of eight lanes cost more than the products of a 16-entry row).
template <int OT, int L, typename F>
__device__ __forceinline__ void ol_product_l(const OlArgs& a, const OlMem& m, int nr, int e0, const double* v, F f) {
    const int lr = threadIdx.x % L, grp = threadIdx.x / L, in_warp = grp % (32 / L);
    const double* __restrict__ vg = a.val + e0;
    for (int base = grp - in_warp; base < nr; base += OT / L) {  // warp-uniform
        const int i = base + in_warp;
        double a0 = 0.0, a1 = 0.0;
        if (i < nr) {
            const int k1 = m.rps[i + 1];
            int k = m.rps[i] + lr;
            if (a.vals_in) {
                for (; k + L < k1; k += 2 * L) {
                    a0 += m.vals[k] * v[m.cols[k]];
                    a1 += m.vals[k + L] * v[m.cols[k + L]];
                }
                if (k < k1) a0 += m.vals[k] * v[m.cols[k]];
            } else {
                for (; k + L < k1; k += 2 * L) {
                    a0 += __ldg(vg + k) * v[m.cols[k]];
                    a1 += __ldg(vg + k + L) * v[m.cols[k + L]];
                }
                if (k < k1) a0 += __ldg(vg + k) * v[m.cols[k]];
            }
        }
        a0 += a1;
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, o, L);
        if (i < nr && lr == 0) f(i, a0);
    }
}
template <int OT, typename F>
__device__ __forceinline__ void ol_product(const OlArgs& a, const OlMem& m, int nr, int e0, const double* v, F f) {
    if (a.lanes == 2) ol_product_l<OT, 2>(a, m, nr, e0, v, f);
    else ol_product_l<OT, 4>(a, m, nr, e0, v, f);
}

// Sums over all rows of the CTAs' arrays u and (TWO) v, one grid barrier: warp 0
// adds u, warp 1 adds v, in a fixed order (FP64 adds by all threads would cost
// more than the barrier).  Valid in every thread through s; false when the
// barrier timed out.
template <bool TWO>
__device__ inline bool ol_sum(const OlArgs& a, GridBarrier& gb, int& slot, const double* u, const double* v, int nr, double* s) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nc = gridDim.x;
    __syncthreads();
    double* part = a.part + (size_t)(slot & 3) * 2 * nc;
    slot += 1;
    if (w < (TWO ? 2 : 1)) {
        const double* z = w ? v : u;
        double t = 0.0, t1 = 0.0;
        int i = lane;
        for (; i + 32 < nr; i += 64) { t += z[i]; t1 += z[i + 32]; }
        if (i < nr) t += z[i];
        t += t1;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) __stcg(part + w * nc + blockIdx.x, t);
    }
    if (!gb.sync()) return false;
    if (w < (TWO ? 2 : 1)) {
        double t = 0.0;
        for (int base = 0; base < nc; base += 160) {
            double p[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int i = base + 32 * k + lane;
                p[k] = i < nc ? __ldcg(part + w * nc + i) : 0.0;
            }
            t += ((p[0] + p[1]) + (p[2] + p[3])) + p[4];
        }
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s[w] = t;
    }
    __syncthreads();
    return true;
}

__device__ inline double ol_dinv(const OlArgs& a, int row) {
    const double d = a.val[a.diag[row]];
    return d != 0.0 ? 1.0 / d : 1.0;
}

// x0 = 0, z = D^-1 r, stop when r.r < tol^2 b.b or after max_iter iterations
template <int OT>
__global__ void __launch_bounds__(OT, OT_CG / OT) k_ol_cg(OlArgs a) {
    extern __shared__ __align__(16) unsigned char ol_smem[];
    __shared__ double s[2], sc;
    __shared__ int ctl;
    GridBarrier gb(a.bar, &a.S->fault, a.bar_start);
    const OlMem m = ol_mem<OT == OT_CG_HALF>(a, ol_smem, 6, 1);
    double *xs = m.row, *rs = xs + a.R, *qs = rs + a.R, *ds = qs + a.R, *w1 = ds + a.R, *w2 = w1 + a.R, *ph = m.hal;
    const int tid = threadIdx.x;
    const int r0 = a.row0[blockIdx.x], nr = a.row0[blockIdx.x + 1] - r0, e0 = a.rp[r0], ne = a.rp[r0 + nr] - e0;
    const int nh = ol_setup<OT>(a, m, r0, nr, e0, ne);
    if (nh > a.H && tid == 0) atomicExch(&a.S->over, 1);
    for (int i = tid; i < nr; i += OT) {
        const double d = ol_dinv(a, r0 + i), r = a.b[r0 + i], z = d * r;
        xs[i] = 0.0;
        ds[i] = d;
        rs[i] = r;
        a.g1[r0 + i] = z;
        w1[i] = r * r;
        w2[i] = r * z;
    }
    int slot = 0;
    if (!ol_sum<true>(a, gb, slot, w1, w2, nr, s)) return;
    if (*(volatile int*)&a.S->over) return;  // the same in every CTA: set before the barrier
    const double bb = s[0], thr = a.tol * a.tol * bb;
    double rz = s[1], rr = bb;
    int iters = 0, fin = !(bb == bb) ? 3 : (bb == 0.0 || bb < thr) ? 1 : 0;
    double beta = 0.0;
    for (int h = tid; h < nh; h += OT) ph[h] = 0.0;
    while (!fin) {
        for (int h = tid; h < nh; h += OT) ph[h] = a.g1[m.hc[h]] + beta * ph[h];
        __syncthreads();
        ol_product<OT>(a, m, nr, e0, ph, [&](int i, double q) {
            qs[i] = q;
            w1[i] = ph[m.li[i]] * q;
        });
        if (!ol_sum<false>(a, gb, slot, w1, w1, nr, s)) return;
        if (tid == 0) sc = rz / s[0];
        __syncthreads();
        const double alpha = sc;
        for (int i = tid; i < nr; i += OT) {
            xs[i] += alpha * ph[m.li[i]];
            const double r = rs[i] - alpha * qs[i], z = ds[i] * r;
            rs[i] = r;
            a.g1[r0 + i] = z;
            w1[i] = r * r;
            w2[i] = r * z;
        }
        if (!ol_sum<true>(a, gb, slot, w1, w2, nr, s)) return;
        rr = s[0];
        iters += 1;
        if (tid == 0) {
            sc = s[1] / rz;
            ctl = (!(s[0] == s[0]) || !(s[1] == s[1])) ? 3 : s[0] < thr ? 1 : iters >= a.max_iter ? 2 : 0;
        }
        rz = s[1];
        __syncthreads();
        beta = sc;
        fin = ctl;
    }
    for (int i = tid; i < nr; i += OT) a.x[r0 + i] = xs[i];
    if (blockIdx.x == 0 && tid == 0) {
        a.S->fin = fin;
        a.S->iters = iters;
        a.S->rr = rr;
        a.S->rhs2 = bb;
    }
}

// fin: 1 converged, 2 iteration limit, 3 breakdown.  When r0.r vanishes, or a
// scalar is not finite, the iteration restarts from the true residual (r0 = r =
// b - A x), as the graph path does for the first of these; a second breakdown
// without an iteration between ends it.
__global__ void __launch_bounds__(OT_BI, 1) k_ol_bicgstab(OlArgs a) {
    constexpr int OT = OT_BI;
    extern __shared__ __align__(16) unsigned char ol_smem[];
    __shared__ double s[2], sc[2];
    __shared__ int ctl;
    GridBarrier gb(a.bar, &a.S->fault, a.bar_start);
    const OlMem m = ol_mem<false>(a, ol_smem, 7, 4);
    double *xs = m.row, *rs = xs + a.R, *r0s = rs + a.R, *vs = r0s + a.R, *ts = vs + a.R, *w1 = ts + a.R, *w2 = w1 + a.R;
    double *ph = m.hal, *dh = ph + a.H, *rh = dh + a.H, *yh = rh + a.H;  // p, D^-1, r, and y or z at the CTA's columns
    const int tid = threadIdx.x;
    const int r0 = a.row0[blockIdx.x], nr = a.row0[blockIdx.x + 1] - r0, e0 = a.rp[r0], ne = a.rp[r0 + nr] - e0;
    const int nh = ol_setup<OT>(a, m, r0, nr, e0, ne);
    if (nh > a.H && tid == 0) atomicExch(&a.S->over, 1);
    for (int i = tid; i < nr; i += OT) {
        const double r = a.b[r0 + i];
        xs[i] = 0.0;
        rs[i] = r0s[i] = r;
        vs[i] = 0.0;
        a.g1[r0 + i] = r;
        a.g2[r0 + i] = 0.0;
        w1[i] = r * r;
    }
    int slot = 0;
    if (!ol_sum<false>(a, gb, slot, w1, w1, nr, s)) return;
    if (*(volatile int*)&a.S->over) return;
    for (int h = tid; h < nh; h += OT) {
        ph[h] = 0.0;
        dh[h] = ol_dinv(a, m.hc[h]);
    }
    const double bb = s[0], tol2 = a.tol * a.tol * bb, eps2 = 2.220446049250313e-16 * 2.220446049250313e-16;
    double rr = bb, rho = bb, alpha = 1.0, w = 1.0, beta = 0.0;  // rho: thread 0 of every CTA
    double *vg = a.g2, *vn = a.g3;                               // v published last, and next
    double r0sq = bb;
    bool rst = false;
    int rst_at = -1;
    int iters = 0, fin = (bb <= tol2 || bb == 0.0) ? 1 : !(bb == bb) ? 3 : 0;
    while (!fin) {
        if (rst) {
            if (rst_at == iters) { fin = 3; break; }
            rst_at = iters;
            rst = false;
            for (int i = tid; i < nr; i += OT) vn[r0 + i] = xs[i];
            if (!gb.sync()) return;
            for (int h = tid; h < nh; h += OT) yh[h] = vn[m.hc[h]];
            __syncthreads();
            ol_product<OT>(a, m, nr, e0, yh, [&](int i, double ax) {
                const double r = a.b[r0 + i] - ax;
                rs[i] = r0s[i] = r;
                a.g1[r0 + i] = r;
                w1[i] = r * r;
            });
            if (!ol_sum<false>(a, gb, slot, w1, w1, nr, s)) return;
            rr = r0sq = rho = s[0];
            alpha = w = 1.0;
            beta = 0.0;
            if (!(rr == rr)) { fin = 3; break; }
            if (rr <= tol2) { fin = 1; break; }
        }
        for (int h = tid; h < nh; h += OT) {
            const int j = m.hc[h];
            const double r = a.g1[j], p = r + beta * (ph[h] - w * vg[j]);
            rh[h] = r;
            ph[h] = p;
            yh[h] = dh[h] * p;
        }
        __syncthreads();
        ol_product<OT>(a, m, nr, e0, yh, [&](int i, double v) {
            vs[i] = v;
            vn[r0 + i] = v;
            w1[i] = r0s[i] * v;
        });
        if (!ol_sum<false>(a, gb, slot, w1, w1, nr, s)) return;
        if (tid == 0) sc[0] = rho / s[0];
        __syncthreads();
        alpha = sc[0];
        if (!(alpha == alpha) || isinf(alpha)) { rst = true; continue; }
        for (int h = tid; h < nh; h += OT) yh[h] = dh[h] * (rh[h] - alpha * vn[m.hc[h]]);  // z = D^-1 s
        __syncthreads();
        ol_product<OT>(a, m, nr, e0, yh, [&](int i, double t) {
            ts[i] = t;
            w1[i] = t * t;
            w2[i] = (rs[i] - alpha * vs[i]) * t;
        });
        if (!ol_sum<true>(a, gb, slot, w1, w2, nr, s)) return;
        if (tid == 0) sc[1] = s[0] > 0.0 ? s[1] / s[0] : 0.0;
        __syncthreads();
        w = sc[1];
        for (int i = tid; i < nr; i += OT) {
            const int l = m.li[i];
            xs[i] += alpha * (dh[l] * ph[l]) + w * yh[l];
            const double r = (rs[i] - alpha * vs[i]) - w * ts[i];
            rs[i] = r;
            a.g1[r0 + i] = r;
            w1[i] = r * r;
            w2[i] = r0s[i] * r;
        }
        if (!ol_sum<true>(a, gb, slot, w1, w2, nr, s)) return;
        rr = s[0];
        iters += 1;
        if (tid == 0) {
            const double trho = s[1];
            int k = 0;
            if (!(s[0] == s[0])) k = 3;
            else if (s[0] <= tol2) k = 1;
            else if (iters >= a.max_iter) k = 2;
            else if (fabs(trho) < eps2 * r0sq) k = 4;
            else {
                sc[0] = (trho / rho) * (alpha / w);
                rho = trho;
                if (!(sc[0] == sc[0]) || isinf(sc[0])) k = 4;
            }
            ctl = k;
        }
        __syncthreads();
        fin = ctl == 4 ? 0 : ctl;
        rst = ctl == 4;
        beta = sc[0];
        double* t = vg;
        vg = vn;
        vn = t;
    }
    for (int i = tid; i < nr; i += OT) a.x[r0 + i] = xs[i];
    if (blockIdx.x == 0 && tid == 0) {
        a.S->fin = fin;
        a.S->iters = iters;
        a.S->rr = rr;
        a.S->rhs2 = bb;
    }
}

// one-launch CG solves in flight, by device
std::atomic<int> ol_running[64];
struct OlRunning {
    std::atomic<int>& n;
    explicit OlRunning(int device) : n(ol_running[device & 63]) { n += 1; }
    ~OlRunning() { n -= 1; }
};

}  // namespace

// FP64 CG (bicg = false) or BiCGSTAB of a system of at most 65,536 equations in
// one launch; *ran = false: it does not fit, or BiCGSTAB broke down (the graph
// path takes over from the start)
int solve_onelaunch(isl_ctx* c, bool bicg, double tol, int64_t max_iter, int64_t* iters, double* rel, bool* nc, bool* ran) {
    *ran = false;
    const int n = (int)c->neq;
    if (c->use_persist != 1 || n == 0 || n > 65536 || (int64_t)c->hrp_small.size() != (int64_t)n + 1) return ISL_OK;
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) != cudaSuccess || !coop) return ISL_OK;
    cudaStream_t st = c->stream;
    const int ncta = std::max(1, std::min(c->sm_count, (n + 31) / 32));
    const std::vector<int32_t>& rp = c->hrp_small;
    // rows balanced by their FP64 work: the stored entries, and about ten
    // operations of the vector updates and sums per row
    std::vector<int32_t> row0((size_t)ncta + 1, n);
    row0[0] = 0;
    int R = 0, E = 0;
    for (int k = 1; k <= ncta; ++k) {
        if (k < ncta) {
            const int64_t goal = ((int64_t)rp[(size_t)n] + 10LL * n) * k / ncta;
            int lo = row0[(size_t)k - 1], hi = n;  // first row whose work before it reaches the goal
            while (lo < hi) {
                const int mid = (lo + hi) / 2;
                if (rp[(size_t)mid] + 10LL * mid < goal) lo = mid + 1;
                else hi = mid;
            }
            row0[(size_t)k] = lo;
        }
        R = std::max(R, row0[(size_t)k] - row0[(size_t)k - 1]);
        E = std::max(E, rp[(size_t)row0[(size_t)k]] - rp[(size_t)row0[(size_t)k - 1]]);
    }
    // the columns of a CTA are not known here: all the room that is left, the
    // values out of shared memory if that leaves too little
    const int nd = bicg ? 7 : 6, nh = bicg ? 4 : 1;
    bool vals = true;
    auto room = [&]() -> int64_t {
        const size_t used = ol_bytes(n, R, E, 0, nd, nh, vals, false);
        return used >= OL_SMEM_MAX ? 0 : (int64_t)(OL_SMEM_MAX - used) / (8 * nh + 4);
    };
    const int64_t want = std::min<int64_t>(n, std::max<int64_t>(4 * (int64_t)R, 1024));
    if (room() < want) vals = false;
    const int64_t H = std::min<int64_t>(n, room());
    if (H < std::min<int64_t>(n, R + 64)) return ISL_OK;
    // beside other solves: with half the shared memory, the values in it or not
    // (how many columns a CTA touches shows in the launch: one that finds too many
    // is done again the next way, and the pattern starts there from then on)
    auto half_columns = [&](bool v) -> int64_t {
        const size_t used = ol_bytes(n, R, E, 0, nd, nh, v, true);
        return used >= OL_SMEM_HALF ? 0 : std::min<int64_t>(n, (int64_t)(OL_SMEM_HALF - used) / (8 * nh + 4));
    };
    const OlRunning running(c->device);
    if (c->ol_half_serial != c->pattern_serial) {
        c->ol_half_serial = c->pattern_serial;
        c->ol_half = 0;
    }
    enum { HALF_VALS = 0, HALF = 1, WHOLE = 2 };
    int form = bicg || running.n == 1 ? WHOLE : c->ol_half;
    if (c->ol_row0.n != row0.size()) ISL_CHECK_CUDA(c, c->ol_row0.alloc(row0.size()));
    if (!c->ol_scal.p) ISL_CHECK_CUDA(c, c->ol_scal.alloc(1));
    if (c->w64.n < (size_t)6 * n) ISL_CHECK_CUDA(c, c->w64.alloc((size_t)6 * n));
    ISL_CHECK_CUDA(c, c->dsol.alloc(n));
    ISL_CHECK_CUDA(c, cudaMemcpyAsync(c->ol_row0.p, row0.data(), row0.size() * 4, cudaMemcpyHostToDevice, st));
    OlArgs a = {n, c->drowptr.p, c->dcolind.p, c->ddiag.p, c->ol_row0.p, c->dval64.p, c->drhs.p, R, E, (int)H, vals ? 1 : 0, c->nnz <= 32 * (int64_t)n ? 2 : 4,
                c->w64.p, c->w64.p + n, c->w64.p + 2 * (size_t)n, c->dsol.p, c->dpart.p, c->dbar.p, 0u, c->ol_scal.p, tol,
                (int)std::min<int64_t>(max_iter, INT32_MAX - 1)};
    OlScal h;
    for (bool done = false; !done;) {
        const bool half = form != WHOLE;
        a.vals_in = form == HALF_VALS || (form == WHOLE && vals);
        a.H = (int)(half ? half_columns(a.vals_in) : H);
        if (half && a.H < std::min<int64_t>(n, R + 64)) { c->ol_half = ++form; continue; }
        const size_t smem = ol_bytes(n, R, E, a.H, nd, nh, a.vals_in, half);
        const void* k = bicg ? (const void*)k_ol_bicgstab : half ? (const void*)k_ol_cg<OT_CG_HALF> : (const void*)k_ol_cg<OT_CG>;
        ISL_CHECK_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OL_SMEM_MAX));
        if (half) ISL_CHECK_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        ISL_CHECK_CUDA(c, grid_barrier_start(c, &a.bar_start));
        ISL_CHECK_CUDA(c, cudaMemsetAsync(c->ol_scal.p, 0, sizeof(OlScal), st));
        void* args[] = {&a};
        ISL_CHECK_CUDA(c, cudaLaunchCooperativeKernel(k, dim3(ncta), dim3(bicg ? OT_BI : half ? OT_CG_HALF : OT_CG), args, smem, st));
        c->launches += 1;
        ISL_CHECK_CUDA(c, cudaMemcpyAsync(&h, c->ol_scal.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        ISL_CHECK_CUDA(c, cudaStreamSynchronize(st));
        done = !half || !h.over;
        if (!done) c->ol_half = ++form;
    }
    if (h.fault) ISL_FAIL(c, ISL_ERR_TIMEOUT, "one-launch FP64 solve: a grid barrier timed out");
    if (h.over || (bicg && h.fin > 2)) return ISL_OK;
    if (h.fin == 3) ISL_FAIL(c, ISL_ERR_NAN, "CG breakdown (non-finite reduction)");
    *ran = true;
    *iters = h.iters;
    *rel = h.rhs2 > 0.0 ? std::sqrt(h.rr / h.rhs2) : 0.0;
    *nc = h.fin == 2;
    return ISL_OK;
}

}  // namespace isl
