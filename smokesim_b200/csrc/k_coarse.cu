// k_coarse.cu - the lower part of the V-cycle (levels Lb..coarsest and back) in
// ONE launch of one thread-block cluster, pressures in shared memory.
//
// As per-level launches these levels cost a launch for each half-sweep (the
// coarsest level alone 2 * n_coarse = 160), at sizes where a launch is all
// latency; in one block the larger of them are bound by the instruction stream
// of one SM (16^3: about 1 us a half-sweep, 24x18x15: 1.3 us); through global
// memory a half-sweep costs an L2 round trip (2 us).  Here
//
//  - a level is cut along its last axis (z, in 2D y) into slabs of planes, one
//    per CTA.  A CTA keeps its slab's pressure in shared memory with one ghost
//    plane on either side, and a thread keeps the weights, divisors and
//    right-hand sides of its cells (at most kCells of each colour) in registers
//    for all sweeps of a visit.  The thread that updates a cell of a slab's end
//    plane also stores it into the neighbour CTA's ghost plane (distributed
//    shared memory); a cluster barrier (about 0.3 us) ends the half-sweep;
//  - a level of at most one cell of each colour per thread of one CTA is solo:
//    CTA 0 runs it alone with block barriers.  A half-sweep is then one
//    dependent chain (barrier, neighbour loads, sum, quotient, store), so it
//    does not branch on the cell - threads without one run the same
//    instructions and drop the store - and only the warps that hold cells take
//    part in the barriers.  The IEEE division's out-of-line path, even where it
//    is never taken, costs that chain about 100 cycles: the quotient is taken
//    from a correctly rounded reciprocal, and where a dividend leaves the range
//    of that form the visit's sweeps are run again with the operator;
//  - pressures lie packed by colour, so consecutive threads read consecutive
//    words: in natural order the stride-2 reads of one colour collide in the
//    banks;
//  - between levels, right-hand sides and coarse pressures go through global
//    memory (L2).
//
// Measured on B200 (one V-cycle, schedule 2 + 2 sweeps, 80 coarsest, whole
// launch): FP32 32^3, 16^3, 8^3 51 us (before: 16^3 and 8^3 in one block from
// shared memory 73 us, and 32^3 as tiled launches 63 us); FP16 storage with the
// response matrix at 128^3 43 us (through global memory 54 us); a coarsest level
// of 24x18x15 cells 85 us (in one block 875 us: 0.5 against 5.4 us a half-sweep).
//
// The arithmetic per cell is that of smooth_cell / residual_cell (a neighbour
// outside the grid is a 0 read from shared memory; its weight still counts in the
// divisor), the restriction's sum order and the prolongation's expression are
// those of k_mg.cu: the same values as the per-level launches, infinities and NaN
// included.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "coarse_level.cuh"
#include "common.cuh"
#include "ss_internal.h"

namespace cg = cooperative_groups;

namespace ss {

constexpr int kThreads = 512;   // 128 registers a thread for two cells of each colour
constexpr int kCells = 2;       // cells of each colour per thread, at most
constexpr int kMaxCtas = 16;
constexpr int kZeros = 32;      // floats of 0, one in each bank, in front of the pressures

// div_recip may take this dividend
SS_D bool recip_ok(float a) {
    const float m = fabsf(a);
    return (m > 1e-25f && m < 1e25f) || __float_as_uint(a) == 0u;
}
// the operator, kept out of the sweeps' instruction stream
__device__ __noinline__ float div_exact(float a, float b) { return a / b; }

struct CoarseLevel {
    int n[3];
    int planes;   // march planes per CTA (solo: all of them)
    int solo;
    int w;        // offset of the slab's pressures in shared memory (floats)
    int tap;      // offset of the axes' prolongation taps (entries)
    float hh, inv_hh;   // h^2 and, where h^2 is a power of two, its exact reciprocal (else 0)
};
template <typename T>
struct CoarseArgs {
    int nlev;
    CoarseLevel lv[SS_MAX_LEVELS];
    T* p[SS_MAX_LEVELS];
    T* r[SS_MAX_LEVELS];
    const float* alpha[SS_MAX_LEVELS];
    int nw, taps, fine;   // floats of the zeros and all pressures; offsets of the tap tables (entries follow) and of the residuals
    int n_pre, n_post, n_coarse, quirks;
    int p_zero;           // the first level's pressure is 0: not read
    float oob_smooth, oob_resid;
    const float* cmat;    // coarsest level by its response matrix (mixed solve), or null: sweeps
    float* cpart;         // the product's slice sums (kProductLanes floats)
};

// One axis position of the prolongation (prolong_pressure.comp:39-51): the
// upper tap's weight and both clamped coarse indices.
struct AxisTap {
    float w;
    unsigned short lo, hi;
};

// One CTA's slab of a level.  ny is 1 in 2D; the march axis m is z (2D: y).
// Packed position q = (m - m0) * ncol + y * hx + (x >> 1) within a colour.
struct Slab {
    int nx, ny, nm, hx, ncol;
    int m0, cnt;      // first plane, cells of a colour (0: none)
    int planes;       // planes of a full slab
    int w[2];         // offset of position 0 per colour (one plane and a word in front of it)
    const AxisTap *tx, *ty, *tm;   // prolongation taps per axis (the last level has none)
    float hh, inv_hh;
};

SS_D float* smf() {
    extern __shared__ float4 smem_coarse[];
    return reinterpret_cast<float*>(smem_coarse);
}

template <int DIM>
SS_HD int slab_floats(const int n[3], int planes) {   // both colours
    const int ncol = (n[0] + 1) / 2 * (DIM == 3 ? n[1] : 1);
    return 2 * ((planes + 2) * ncol + 2);
}

template <int DIM, typename T>
SS_D Slab slab_of(const CoarseArgs<T>& b, int l, int rank) {
    const CoarseLevel& v = b.lv[l];
    Slab g;
    g.nx = v.n[0];
    g.ny = DIM == 3 ? v.n[1] : 1;
    g.nm = DIM == 3 ? v.n[2] : v.n[1];
    g.hx = (g.nx + 1) >> 1;
    g.ncol = g.hx * g.ny;
    g.planes = v.planes;
    g.m0 = v.solo ? 0 : rank * v.planes;
    const int have = v.solo ? (rank == 0 ? g.nm : 0) : max(0, min(v.planes, g.nm - g.m0));
    g.cnt = have * g.ncol;
    const int colour = (v.planes + 2) * g.ncol + 2;
    g.w[0] = v.w + g.ncol + 1;
    g.w[1] = g.w[0] + colour;
    g.tx = reinterpret_cast<const AxisTap*>(smf() + b.taps) + v.tap;
    g.ty = g.tx + g.nx;
    g.tm = DIM == 3 ? g.ty + g.ny : g.ty;
    g.hh = v.hh;
    g.inv_hh = v.inv_hh;
    return g;
}

// a thread's cells of a slab: per colour and cell the fluid weights (0 outside
// the grid), their sum and its reciprocal under the smoother's rule, their sum
// under the residual's, and the right-hand side
template <int K>
struct Cells {
    float f[2][K][6], fs[2][K], yr[2][K], fr[2][K], r[2][K];
    int x2[K], y[K], m[K];   // the pair's even x, its row and plane
    int odd[K];              // x parity of the red cell (the black one's is the other)
    int nb[2][K][6];         // the neighbours' places in shared memory (outside the grid: one of the zeros)
    bool act[2][K];          // updated by the sweeps
    bool live[2][K];         // not solid
    bool in[2][K];           // a cell of the grid
    SS_D int x(int k, int j) const { return x2[j] + (odd[j] ^ k); }
    SS_D int index(const Slab& g, int k, int j) const { return (m[j] * g.ny + y[j]) * g.nx + x(k, j); }
};

// Every load is issued before the first is used: one memory latency a visit.
template <int DIM, int K, typename T>
SS_D void load_cells(const Slab& g, const float* __restrict__ alpha, const T* r, float oob_s, float oob_r, Cells<K>& c) {
    float a[2][K][7];
    T rr[2][K];
    auto edges = [&](int k, int j, bool e[6]) {
        e[0] = DIM == 3 ? c.y[j] + 1 < g.ny : c.m[j] + 1 < g.nm;
        e[1] = DIM == 3 ? c.y[j] > 0 : c.m[j] > 0;
        e[2] = c.x(k, j) + 1 < g.nx;
        e[3] = c.x(k, j) > 0;
        e[4] = DIM == 3 && c.m[j] + 1 < g.nm;
        e[5] = DIM == 3 && c.m[j] > 0;
    };
    // A neighbour outside the grid is read as 0, from a bank that no other lane reads:
    // no test in the sweeps and no bank conflict.  Past the end of a row that is the
    // bank of the row's other end: that of its place in the packed order is the next
    // row's, whose lane may be reading there (8^3: 7 cycles more of 207 a half-sweep).
    // In 3D the places are formed after the loads are issued (reverse pass of a 64^3
    // solve of 8 V-cycles 1661 us, 1708 before them), in 2D before them (8 V-cycles at
    // 256^2 with 16-bit storage 511 us; 559 after them, where those forms spill).
    auto places = [&](int k, int j) {
        bool e[6];
        edges(k, j, e);
        const int at = (k ? g.w[0] : g.w[1]) + threadIdx.x + j * kThreads, right = c.odd[j] ^ k, ts = DIM == 3 ? g.hx : g.ncol;
        auto place = [&](int to, bool inside) { return (at + to) & (c.in[k][j] && inside ? -1 : kZeros - 1); };
        int* nb = c.nb[k][j];
        nb[0] = place(ts, e[0]);
        nb[1] = place(-ts, e[1]);
        nb[2] = place(e[2] ? right : right - g.hx, e[2]);
        nb[3] = place(e[3] ? right - 1 : right - 1 + g.hx, e[3]);
        if constexpr (DIM == 3) {
            nb[4] = place(g.ncol, e[4]);
            nb[5] = place(-g.ncol, e[5]);
        }
    };
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int q = threadIdx.x + j * kThreads, pl = q / g.ncol, col = q - pl * g.ncol, y = col / g.hx;
        c.x2[j] = 2 * (col - y * g.hx);
        c.y[j] = y;
        c.m[j] = g.m0 + pl;
        c.odd[j] = (y + c.m[j]) & 1;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            c.in[k][j] = q < g.cnt && c.x(k, j) < g.nx;
            const int i = c.index(g, k, j), off[6] = {g.nx, -g.nx, 1, -1, g.nx * g.ny, -g.nx * g.ny};
            if constexpr (DIM == 2) places(k, j);
            bool e[6];
            edges(k, j, e);
            a[k][j][6] = 1.f;
            if (c.in[k][j]) {
                a[k][j][6] = __ldg(alpha + i);
                rr[k][j] = __ldcg(r + i);
            }
#pragma unroll
            for (int d = 0; d < 6; ++d) a[k][j][d] = c.in[k][j] && e[d] ? __ldg(alpha + i + off[d]) : 1.f;
        }
    }
    if constexpr (DIM == 3)
#pragma unroll
        for (int j = 0; j < K; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) places(k, j);
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float* f = c.f[k][j];
            c.fs[k][j] = c.yr[k][j] = c.fr[k][j] = 1.f;
            c.r[k][j] = 0.f;
            c.act[k][j] = c.live[k][j] = false;
#pragma unroll
            for (int d = 0; d < 6; ++d) f[d] = 1.f - a[k][j][d];
            if (!c.in[k][j]) continue;
            c.r[k][j] = ld(rr[k][j]);
            bool e[6];
            edges(k, j, e);
            // the divisors count an out-of-grid neighbour as 1 - oob
            auto total = [&](float o) {
                float s = (e[0] ? f[0] : o) + (e[1] ? f[1] : o) + (e[2] ? f[2] : o) + (e[3] ? f[3] : o);
                if constexpr (DIM == 3) s = s + (e[4] ? f[4] : o) + (e[5] ? f[5] : o);
                return s;
            };
            c.fr[k][j] = total(1.f - oob_r);
            const float fs = total(1.f - oob_s);
            c.live[k][j] = a[k][j][6] < 1.f;
            c.act[k][j] = c.live[k][j] && fs != 0.f;
            if (c.act[k][j]) {
                c.fs[k][j] = fs;
                c.yr[k][j] = 1.f / fs;
            }
        }
}

// neighbour sum of cell j of colour k, in smooth_cell's order
template <int DIM, int K>
SS_D float cell_sum(const Cells<K>& c, int k, int j) {
    const float* P = smf();
    const float* f = c.f[k][j];
    const int* nb = c.nb[k][j];
    float s = P[nb[0]] * f[0] + P[nb[1]] * f[1];
    s = s + P[nb[2]] * f[2];
    s = s + P[nb[3]] * f[3];
    if constexpr (DIM == 3) {
        s = s + P[nb[4]] * f[4];
        s = s + P[nb[5]] * f[5];
    }
    return s;
}

// barrier over the first nt threads of the block (nt a multiple of 32)
SS_D void sync_first(int nt) {
    if (nt == 32) __syncwarp();
    else if (nt == kThreads) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
}

// stores of end-plane cells into the neighbour CTAs' ghost planes
struct Ghosts {
    float *below, *above;   // shared memory of the CTAs with the planes below and above, or null
    int span;               // cells of a full slab
    SS_D Ghosts(cg::cluster_group* cl, const Slab& g, int rank) {
        below = cl && g.cnt > 0 && g.m0 > 0 ? cl->map_shared_rank(smf(), rank - 1) : nullptr;
        above = cl && g.cnt > 0 && g.m0 + g.planes < g.nm ? cl->map_shared_rank(smf(), rank + 1) : nullptr;
        span = g.planes * g.ncol;
    }
    SS_D void push(const Slab& g, int k, int q, float v) const {
        const int w = (k ? g.w[1] : g.w[0]) + q;
        if (below && q < g.ncol) below[w + span] = v;
        if (above && q >= span - g.ncol) above[w - span] = v;
    }
};

// red-black sweeps of a slab that all CTAs run together
template <int DIM, typename R, int K>
SS_D void split_sweeps(cg::cluster_group& cl, const Slab& g, const Cells<K>& c, int iterations, const Ghosts& gh) {
    float* F = smf();
    for (int it = 0; it < iterations; ++it) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float v[K];
#pragma unroll
            for (int j = 0; j < K; ++j) v[j] = cell_sum<DIM>(c, k, j) - c.r[k][j] * g.hh;
#pragma unroll
            for (int j = 0; j < K; ++j) {
                float q = div_recip(v[j], c.fs[k][j], c.yr[k][j]);
                if (!recip_ok(v[j])) q = div_exact(v[j], c.fs[k][j]);
                q = rnd<R>(q);
                if (c.act[k][j]) {
                    const int at = threadIdx.x + j * kThreads;
                    F[(k ? g.w[1] : g.w[0]) + at] = q;
                    gh.push(g, k, at, q);
                }
            }
            cl.sync();
        }
    }
}

template <int DIM, typename R, int K, bool EXACT>
SS_D bool solo_loop(const Slab& g, const Cells<K>& c, int iterations, int nt) {
    float* F = smf();
    bool ok = true;
    for (int it = 0; it < iterations; ++it) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float v[K];
#pragma unroll
            for (int j = 0; j < K; ++j) v[j] = cell_sum<DIM>(c, k, j) - (c.act[k][j] ? c.r[k][j] * g.hh : -1.f);
#pragma unroll
            for (int j = 0; j < K; ++j) {
                const float q = EXACT ? div_exact(v[j], c.fs[k][j]) : div_recip(v[j], c.fs[k][j], c.yr[k][j]);
                if (!EXACT) ok = ok && recip_ok(v[j]);
                if (c.act[k][j]) F[(k ? g.w[1] : g.w[0]) + threadIdx.x + j * kThreads] = rnd<R>(q);
            }
            sync_first(nt);
        }
    }
    return ok;
}

// red-black sweeps of a solo level by CTA 0
template <int DIM, typename R, int K>
SS_D void solo_sweeps(const Slab& g, const Cells<K>& c, int iterations) {
    float* F = smf();
    const int nt = min(kThreads, (g.cnt + 31) & ~31);
    const bool part = (int)threadIdx.x < nt;
    float p0[2][K];
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) p0[k][j] = c.act[k][j] ? F[(k ? g.w[1] : g.w[0]) + threadIdx.x + j * kThreads] : 0.f;
    __syncthreads();
    bool ok = true;
    if (part) ok = solo_loop<DIM, R, K, false>(g, c, iterations, nt);
    if (__syncthreads_and(ok)) return;
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (c.act[k][j]) F[(k ? g.w[1] : g.w[0]) + threadIdx.x + j * kThreads] = p0[k][j];
    __syncthreads();
    if (part) solo_loop<DIM, R, K, true>(g, c, iterations, nt);
    __syncthreads();
}

// residuals of a slab (restrict_residual reads them from `fine`, packed like the
// pressures without ghosts); with the reference's rule also over r
template <int DIM, typename R, int K, typename T>
SS_D void slab_residual(const Slab& g, const Cells<K>& c, int fine, bool quirks, T* r) {
    float* F = smf();
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!c.in[k][j]) continue;
            const int q = threadIdx.x + j * kThreads;
            const float lap = cell_sum<DIM>(c, k, j) - c.fr[k][j] * F[(k ? g.w[1] : g.w[0]) + q];
            float res = c.r[k][j] - (g.inv_hh != 0.f ? lap * g.inv_hh : lap / g.hh);
            if (!c.live[k][j]) res = 0.f;
            if (quirks) {
                res = rnd<R>(res);
                r[c.index(g, k, j)] = st<T>(res);
            }
            F[fine + k * g.planes * g.ncol + q] = res;
        }
}

// this CTA's share of the next level's right-hand side; the fine residuals
// are those of all CTAs (cl: the cluster, where the fine level is split)
template <int DIM, typename R, typename T>
SS_D void restrict_share(cg::cluster_group* cl, const Slab& g, int fine, const int cn[3], T* rc, int rank, int ctas) {
    const int cx = cn[0], cy = DIM == 3 ? cn[1] : 1, cm = DIM == 3 ? cn[2] : cn[1], n = cx * cy * cm;
    const int share = cl ? ctas : 1;
    for (int i = (cl ? rank : 0) * kThreads + threadIdx.x; i < n; i += share * kThreads) {
        const int X = i % cx, t = i / cx, Y = t % cy, M = t / cy;
        auto v = [&](int dx, int dy, int dm) {
            const int y = DIM == 3 ? 2 * Y + dy : 0, m = 2 * M + dm, owner = m / g.planes;
            const int k = (dx + y + m) & 1;
            const float* at = smf() + fine + k * g.planes * g.ncol + (m - owner * g.planes) * g.ncol + y * g.hx + X;
            return cl ? *cl->map_shared_rank(at, owner) : *at;
        };
        float out;
        if constexpr (DIM == 3) {
            const float bottom = v(0, 0, 0) + v(0, 0, 1) + v(1, 0, 0) + v(1, 0, 1);
            const float top = v(0, 1, 0) + v(0, 1, 1) + v(1, 1, 0) + v(1, 1, 1);
            out = (bottom + top) / 8.f;
        } else {
            out = (v(0, 0, 0) + v(1, 0, 0) + v(0, 0, 1) + v(1, 0, 1)) / 4.f;
        }
        rc[i] = st<T>(rnd<R>(out));
    }
}

// Prolongation: the coarse planes the slab reads come into shared memory once
// (the residuals' place), then every cell adds its interpolated correction.
template <int DIM, typename R, int K, typename T>
SS_D void slab_prolong(const Slab& g, const Cells<K>& c, const int cn[3], const T* pc, int stage, const Ghosts& gh) {
    float* F = smf();
    const int cx = cn[0], cy = DIM == 3 ? cn[1] : 1;
    if (g.cnt == 0) {
        __syncthreads();
        return;
    }
    const int lo = g.tm[g.m0].lo, hi = g.tm[g.m0 + g.cnt / g.ncol - 1].hi, n = (hi - lo + 1) * cx * cy;
    const T* src = pc + lo * cx * cy;
    for (int i = threadIdx.x; i < n; i += 4 * kThreads) {
        T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * kThreads < n) v[u] = __ldcg(src + i + u * kThreads);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * kThreads < n) F[stage + i + u * kThreads] = ld(v[u]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!c.in[k][j]) continue;
            const int q = threadIdx.x + j * kThreads;
            const AxisTap X = g.tx[c.x(k, j)], M = g.tm[c.m[j]];
            const float* A = F + stage;
            float s;
            if constexpr (DIM == 2) {
                const float *a = A + (M.lo - lo) * cx, *d = A + (M.hi - lo) * cx;
                s = lerp_(lerp_(a[X.lo], a[X.hi], X.w), lerp_(d[X.lo], d[X.hi], X.w), M.w);
            } else {
                const AxisTap Y = g.ty[c.y[j]];
                const float *a = A + ((M.lo - lo) * cy + Y.lo) * cx, *d = A + ((M.lo - lo) * cy + Y.hi) * cx;
                const float *e = A + ((M.hi - lo) * cy + Y.lo) * cx, *h = A + ((M.hi - lo) * cy + Y.hi) * cx;
                const float c0 = lerp_(lerp_(a[X.lo], a[X.hi], X.w), lerp_(d[X.lo], d[X.hi], X.w), Y.w);
                const float c1 = lerp_(lerp_(e[X.lo], e[X.hi], X.w), lerp_(h[X.lo], h[X.hi], X.w), Y.w);
                s = lerp_(c0, c1, M.w);
            }
            float* P = F + (k ? g.w[1] : g.w[0]) + q;
            const float v = rnd<R>(*P + s);
            *P = v;
            gh.push(g, k, q, v);
        }
}

template <int DIM, int K, typename T>
SS_D void slab_store(const Slab& g, const Cells<K>& c, T* p) {
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!c.in[k][j]) continue;
            p[c.index(g, k, j)] = st<T>(smf()[(k ? g.w[1] : g.w[0]) + threadIdx.x + j * kThreads]);
        }
}

// One visit of level l by this CTA: up = 0 on the way down (pre-smoothing,
// residual, restriction; the coarsest level's sweeps), 1 on the way up
// (prolongation, post-smoothing).  cl: the cluster on a split level, else null.
template <int DIM, typename T, typename R, int K>
SS_D void visit(const CoarseArgs<T>& b, int l, bool up, cg::cluster_group* cl, int rank, int ctas) {
    const Slab g = slab_of<DIM>(b, l, rank);
    Cells<K> c;
    load_cells<DIM>(g, b.alpha[l], b.r[l], b.oob_smooth, b.oob_resid, c);
    const Ghosts gh(cl, g, rank);
    const bool last = l == b.nlev - 1;
    auto sync = [&]() {
        if (cl) cl->sync();
        else __syncthreads();
    };
    if (!up && l == 0 && !b.p_zero) {
#pragma unroll
        for (int j = 0; j < K; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (!c.in[k][j]) continue;
                const int q = threadIdx.x + j * kThreads;
                const float v = ld(b.p[0][c.index(g, k, j)]);
                smf()[(k ? g.w[1] : g.w[0]) + q] = v;
                gh.push(g, k, q, v);
            }
        sync();
    }
    if (up) {
        slab_prolong<DIM, R>(g, c, b.lv[l + 1].n, b.p[l + 1], b.fine, gh);
        sync();
    }
    const int sweeps = up ? b.n_post : last ? b.n_coarse : b.n_pre;
    if (cl) split_sweeps<DIM, R>(*cl, g, c, sweeps, gh);
    else solo_sweeps<DIM, R>(g, c, sweeps);
    if (up || last) {
        slab_store<DIM>(g, c, b.p[l]);
        return;
    }
    slab_residual<DIM, R>(g, c, b.fine, b.quirks != 0, b.r[l]);
    sync();
    restrict_share<DIM, R>(cl, g, b.fine, b.lv[l + 1].n, b.r[l + 1], rank, ctas);
}

// the axes' prolongation taps, which depend on the sizes alone
template <int DIM, typename T>
SS_D void build_taps(const CoarseArgs<T>& b) {
    for (int l = 0; l + 1 < b.nlev; ++l) {
        AxisTap* tap = reinterpret_cast<AxisTap*>(smf() + b.taps) + b.lv[l].tap;
        const int nx = b.lv[l].n[0], ny = b.lv[l].n[1], nz = b.lv[l].n[2];
        for (int i = threadIdx.x; i < nx + ny + (DIM == 3 ? nz : 0); i += kThreads) {
            const int d = i < nx ? 0 : i < nx + ny ? 1 : 2, at = i - (d > 0 ? nx : 0) - (d > 1 ? ny : 0);
            const int a = b.lv[l].n[d], c = b.lv[l + 1].n[d];
            const float t = (((float)at + 0.5f) / (float)a) * (float)c - 0.5f;
            const float f = floorf(t);
            AxisTap v;
            v.w = t - f;
            v.lo = (unsigned short)min(max((int)f, 0), c - 1);
            v.hi = (unsigned short)min(max((int)f + 1, 0), c - 1);
            tap[i] = v;
        }
    }
}

template <int DIM, typename T, typename R>
__global__ void __launch_bounds__(kThreads) k_coarse(const __grid_constant__ CoarseArgs<T> b) {
    cg::cluster_group cl = cg::this_cluster();
    const int ctas = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    float* F = smf();
    // pressures and ghost planes start at 0 (the initial guess, and the pressure
    // outside the grid); every CTA has done so before a neighbour stores here
    for (int i = threadIdx.x; i < b.nw; i += kThreads) F[i] = 0.f;
    build_taps<DIM>(b);
    cl.sync();
    pdl_entry();
    // The level-0 sweeps since the last V-cycle have pushed the lower levels'
    // arrays out of L2 on large grids: their lines come back while the first
    // level is at work, instead of one visit after the other.
    auto prefetch = [&](const void* p, long long bytes) {
        for (long long i = ((long long)rank * kThreads + threadIdx.x) * 128; i < bytes; i += (long long)ctas * kThreads * 128)
            prefetch_l2(reinterpret_cast<const char*>(p) + i);
    };
    for (int l = 1; l < b.nlev; ++l) prefetch(b.alpha[l], 4LL * b.lv[l].n[0] * b.lv[l].n[1] * b.lv[l].n[2]);
    if (b.cmat) {
        const long long n = (long long)b.lv[b.nlev - 1].n[0] * b.lv[b.nlev - 1].n[1] * b.lv[b.nlev - 1].n[2];
        prefetch(b.cmat, 4 * n * n);
    }
    auto run = [&](int l, bool up) {
        const CoarseLevel& v = b.lv[l];
        if (v.solo && rank != 0) return;
        const int ncol = (v.n[0] + 1) / 2 * (DIM == 3 ? v.n[1] : 1);
        const bool two = v.planes * ncol > kThreads;
        if (two) visit<DIM, T, R, 2>(b, l, up, v.solo ? nullptr : &cl, rank, ctas);
        else visit<DIM, T, R, 1>(b, l, up, v.solo ? nullptr : &cl, rank, ctas);
    };
    // between two visits: CTA 0 alone where both levels are solo
    auto between = [&](int l0, int l1) {
        if (b.lv[l0].solo && b.lv[l1].solo) __syncthreads();
        else cl.sync();
    };
    const int last = b.nlev - 1;
    for (int l = 0; l < last; ++l) {
        run(l, false);
        if (l + 1 < last || !b.cmat) between(l, l + 1);
    }
    if (b.cmat) {
        const int n = b.lv[last].n[0] * b.lv[last].n[1] * b.lv[last].n[2];
        cl.sync();
        for (int i = threadIdx.x; i < n; i += kThreads) F[b.fine + i] = ld(__ldcg(b.r[last] + i));
        __syncthreads();
        coarse_matrix_partials(b.cmat, F + b.fine, b.cpart, n, rank * kThreads + (int)threadIdx.x, ctas * kThreads);
        cl.sync();
        coarse_matrix_fold<R>(b.cpart, b.p[last], n, rank * kThreads + (int)threadIdx.x, ctas * kThreads);
        cl.sync();
    } else {
        run(last, false);
        if (last > 0) between(last, last - 1);
    }
    for (int l = last - 1; l >= 0; --l) {
        run(l, true);
        if (l > 0) between(l, l - 1);
    }
    cl.sync();   // no CTA leaves while its shared memory may be read or written
}

// ------------------------------------------------------------- the transpose
// The lower V-cycle's transpose (levels Lb..coarsest and back) over the same
// slabs.  p is the adjoint of the levels' pressures, r that of their right-hand
// sides (both natural, global); a thread keeps its cells' values of both in
// registers through a visit's sweeps, and shared memory holds T, the quotient
// each transposed update passes to its neighbours (k_adj_smooth in
// k_adjoint.cu has the operator).  One visit is bound by its cluster barriers
// and L2 round trips: 32^3, 16^3 and 8^3 with the response matrix take 54 us,
// against 66 for the last two in one block and 21 launches and copies for 32^3.
template <int DIM, int K>
SS_D void adj_sweeps_slab(cg::cluster_group* cl, const Slab& g, const Cells<K>& c, const float (&ws)[2][K],
                          float (&pb)[2][K], float (&bb)[2][K], int iterations, const Ghosts& gh) {
    float* F = smf();
    for (int it = 0; it < iterations; ++it) {
#pragma unroll
        for (int k = 1; k >= 0; --k) {
            // the gather half of the colour before (none before the first), then this colour's transpose
            float v[K];
#pragma unroll
            for (int j = 0; j < K; ++j)
                v[j] = it == 0 && k == 1 ? pb[k][j] : pb[k][j] + ws[k][j] * cell_sum<DIM>(c, k, j);
#pragma unroll
            for (int j = 0; j < K; ++j) {
                float t = div_recip(v[j], c.fs[k][j], c.yr[k][j]);
                if (!recip_ok(v[j])) t = div_exact(v[j], c.fs[k][j]);
                if (c.act[k][j]) {
                    const int at = threadIdx.x + j * kThreads;
                    F[(k ? g.w[1] : g.w[0]) + at] = t;
                    gh.push(g, k, at, t);
                    bb[k][j] -= g.hh * t;
                }
                pb[k][j] = c.act[k][j] ? 0.f : v[j];
            }
            if (cl) cl->sync();
            else __syncthreads();
        }
    }
    if (iterations > 0)
#pragma unroll
        for (int j = 0; j < K; ++j) pb[1][j] += ws[1][j] * cell_sum<DIM>(c, 1, j);
}

// One visit of level l: on the way down the post-smoothing's transpose (the
// coarsest level's sweeps), on the way up that of residual, restriction and
// pre-smoothing.
template <int DIM, int K>
SS_D void adj_visit(const CoarseArgs<float>& b, int l, bool up, cg::cluster_group* cl, int rank) {
    const Slab g = slab_of<DIM>(b, l, rank);
    const bool last = l == b.nlev - 1;
    Cells<K> c;
    load_cells<DIM>(g, b.alpha[l], b.alpha[l], b.oob_smooth, b.oob_resid, c);   // c.r: the cell's own alpha
    float ws[2][K], pb[2][K], bb[2][K];
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            ws[k][j] = c.in[k][j] ? 1.f - c.r[k][j] : 0.f;
            pb[k][j] = c.in[k][j] ? __ldcg(b.p[l] + c.index(g, k, j)) : 0.f;
            bb[k][j] = up && c.in[k][j] ? __ldcg(b.r[l] + c.index(g, k, j)) : 0.f;
        }
    if (up) {
        const int cx = b.lv[l + 1].n[0], cy = DIM == 3 ? b.lv[l + 1].n[1] : 1, cm = b.lv[l + 1].n[DIM == 3 ? 2 : 1];
        auto parent = [&](int x, int y, int m) -> float {   // the residual's adjoint at a fluid cell
            const int X = x >> 1, Y = DIM == 3 ? y >> 1 : 0, M = m >> 1;
            return X < cx && Y < cy && M < cm ? __ldcg(b.r[l + 1] + (M * cy + Y) * cx + X) * (DIM == 3 ? 0.125f : 0.25f) : 0.f;
        };
#pragma unroll
        for (int j = 0; j < K; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (!c.in[k][j]) continue;
                const float* f = c.f[k][j];   // 0: solid or out of grid
                const int x = c.x(k, j), y = c.y[j], m = c.m[j];
                const float rs = c.live[k][j] ? parent(x, y, m) : 0.f;
                float nb = 0.f;
                if (f[0] > 0.f) nb += DIM == 3 ? parent(x, y + 1, m) : parent(x, y, m + 1);
                if (f[1] > 0.f) nb += DIM == 3 ? parent(x, y - 1, m) : parent(x, y, m - 1);
                if (f[2] > 0.f) nb += parent(x + 1, y, m);
                if (f[3] > 0.f) nb += parent(x - 1, y, m);
                if constexpr (DIM == 3) {
                    if (f[4] > 0.f) nb += parent(x, y, m + 1);
                    if (f[5] > 0.f) nb += parent(x, y, m - 1);
                }
                pb[k][j] += (c.fr[k][j] * rs - ws[k][j] * nb) / g.hh;
                bb[k][j] += rs;
            }
    }
    // the gather takes its neighbours' T unweighted; a solid neighbour's is 0
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int d = 0; d < 6; ++d) c.f[k][j][d] = c.f[k][j][d] > 0.f ? 1.f : 0.f;
    const Ghosts gh(cl, g, rank);
    adj_sweeps_slab<DIM>(cl, g, c, ws, pb, bb, up ? b.n_pre : last ? b.n_coarse : b.n_post, gh);
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!c.in[k][j]) continue;
            if (!up) b.p[l][c.index(g, k, j)] = pb[k][j];
            b.r[l][c.index(g, k, j)] = bb[k][j];
        }
}

// Transpose of the prolongation onto level l (k_adj_prolong's sums), by all
// threads of the cluster: the fine window of coarse index K is [2K-2, 2K+3].
template <int DIM>
SS_D void adj_prolong_share(const CoarseArgs<float>& b, int l, int first, int threads) {
    const int* cn = b.lv[l].n;
    const int* fn = b.lv[l - 1].n;
    const AxisTap* tap = reinterpret_cast<const AxisTap*>(smf() + b.taps) + b.lv[l - 1].tap;
    const int n = cn[0] * cn[1] * (DIM == 3 ? cn[2] : 1);
    for (int i = first; i < n; i += threads) {
        const int X = i % cn[0], t = i / cn[0], Y = t % cn[1], Z = t / cn[1];
        auto coef = [&](int d, int x, int K) -> float {
            if (x < 0 || x >= fn[d]) return 0.f;
            const AxisTap v = tap[x + (d > 0 ? fn[0] : 0) + (d > 1 ? fn[1] : 0)];
            return (v.lo == K ? 1.f - v.w : 0.f) + (v.hi == K ? v.w : 0.f);
        };
        float wx[6], wy[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            wx[q] = coef(0, 2 * X - 2 + q, X);
            wy[q] = coef(1, 2 * Y - 2 + q, Y);
        }
        float s = 0.f;
        for (int k = 0; k < (DIM == 3 ? 6 : 1); ++k) {
            const int z = DIM == 3 ? 2 * Z - 2 + k : 0;
            const float wz = DIM == 3 ? coef(2, z, Z) : 1.f;
            if (wz == 0.f) continue;
            float v[6][6];
#pragma unroll
            for (int j = 0; j < 6; ++j)
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    v[j][q] = wy[j] != 0.f && wx[q] != 0.f
                                  ? __ldcg(b.p[l - 1] + (z * fn[1] + 2 * Y - 2 + j) * fn[0] + 2 * X - 2 + q) : 0.f;
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                float row = 0.f;
#pragma unroll
                for (int q = 0; q < 6; ++q) row += wx[q] * v[j][q];
                s += wz * wy[j] * row;
            }
        }
        b.p[l][i] = s;
    }
}

template <int DIM>
__global__ void __launch_bounds__(kThreads) k_adj_coarse(const __grid_constant__ CoarseArgs<float> b) {
    cg::cluster_group cl = cg::this_cluster();
    const int ctas = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int first = rank * kThreads + (int)threadIdx.x, threads = ctas * kThreads;
    float* F = smf();
    for (int i = threadIdx.x; i < b.nw; i += kThreads) F[i] = 0.f;   // T outside the grid and of solid cells
    build_taps<DIM>(b);
    cl.sync();
    auto run = [&](int l, bool up) {
        const CoarseLevel& v = b.lv[l];
        if (!v.solo || rank == 0) {
            const int ncol = (v.n[0] + 1) / 2 * (DIM == 3 ? v.n[1] : 1);
            if (v.planes * ncol > kThreads) adj_visit<DIM, 2>(b, l, up, v.solo ? nullptr : &cl, rank);
            else adj_visit<DIM, 1>(b, l, up, v.solo ? nullptr : &cl, rank);
        }
        cl.sync();
    };
    const int last = b.nlev - 1;
    for (int l = 0; l < last; ++l) {
        run(l, false);
        adj_prolong_share<DIM>(b, l + 1, first, threads);
        cl.sync();
    }
    if (b.cmat) {
        // the coarsest sweeps as one product: r = D^T p, D[j n + i] = dp_j / dr_i
        const int n = b.lv[last].n[0] * b.lv[last].n[1] * b.lv[last].n[2];
        for (int i = threadIdx.x; i < n; i += kThreads) F[b.fine + i] = __ldcg(b.p[last] + i);
        __syncthreads();
        coarse_matrix_partials(b.cmat, F + b.fine, b.cpart, n, first, threads);
        cl.sync();
        coarse_matrix_fold<float>(b.cpart, b.r[last], n, first, threads);
        cl.sync();
    } else {
        run(last, false);
    }
    for (int l = last - 1; l >= 0; --l) run(l, true);
}

// ------------------------------------------------------------------ host
static bool pow2_normal(float v) {
    if (!(v > 0.f) || !std::isfinite(v)) return false;
    int e;
    return std::frexp(v, &e) == 0.5f && v >= 1.1754944e-38f && v <= 1e30f;
}

static int level_ncol(const ss_sim* s, int l) { return (s->lv[l].n[0] + 1) / 2 * (s->dim == 3 ? s->lv[l].n[1] : 1); }
static int level_nm(const ss_sim* s, int l) { return s->dim == 3 ? s->lv[l].n[2] : s->lv[l].n[1]; }

// planes per CTA of level l on `ctas` CTAs, 0 where it does not fit; *solo: CTA 0 alone
static int level_planes(const ss_sim* s, int l, int ctas, int* solo) {
    const int ncol = level_ncol(s, l), nm = level_nm(s, l);
    *solo = ctas == 1 || (long long)ncol * nm <= kThreads;
    const int planes = *solo ? nm : (nm + ctas - 1) / ctas;
    return (long long)planes * ncol <= kCells * kThreads ? planes : 0;
}

// shared memory in floats of levels L.. on `ctas` CTAs: zeros, pressures, prolongation
// taps, then the residuals / staged coarse planes / the matrix product's vector
static long long coarse_floats(const ss_sim* s, int L, int ctas, long long* nw, long long* ntap) {
    long long w = kZeros, taps = 0, fine = 0;
    for (int l = L; l < s->levels; ++l) {
        int solo;
        const int planes = level_planes(s, l, ctas, &solo);
        if (!planes) return -1;
        const int* n = s->lv[l].n;
        w += s->dim == 3 ? slab_floats<3>(n, planes) : slab_floats<2>(n, planes);
        taps += n[0] + n[1] + (s->dim == 3 ? n[2] : 0);
        fine = std::max(fine, 2LL * planes * level_ncol(s, l));
        if (l + 1 < s->levels) {
            // coarse planes under `planes` fine ones: one more than half on either side
            const int* c = s->lv[l + 1].n;
            const int cm = s->dim == 3 ? c[2] : c[1];
            fine = std::max(fine, (long long)std::min(cm, planes / 2 + 3) * c[0] * (s->dim == 3 ? c[1] : 1));
        } else {
            fine = std::max(fine, (long long)n[0] * n[1] * n[2] <= kCoarseResponseMax ? (long long)n[0] * n[1] * n[2] : 0LL);
        }
    }
    *nw = (w + 1) & ~1LL;   // the taps are 8-byte entries
    *ntap = taps;
    return *nw + 2 * taps + fine;
}

constexpr long long kCoarseSmem = 200 * 1024;

// The smallest cluster (a power of two of at most max_ctas CTAs) on which
// levels L.. fit; 0: none.  On one with a single cell of each colour per thread
// of the first level where there is such a one.
static int coarse_ctas(const ss_sim* s, int L, int max_ctas) {
    int fits = 0;
    for (int c = 1; c <= max_ctas; c *= 2) {
        long long nw, taps;
        const long long f = coarse_floats(s, L, c, &nw, &taps);
        if (f < 0 || f * (long long)sizeof(float) > kCoarseSmem) continue;
        int solo;
        fits = c;
        if ((long long)level_planes(s, L, c, &solo) * level_ncol(s, L) <= kThreads) break;
    }
    return fits;
}

static void coarse_config(int ctas, size_t smem, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3(ctas);
    cfg->blockDim = dim3(kThreads);
    cfg->dynamicSmemBytes = smem;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}

template <typename K>
static cudaError_t coarse_attributes(K* kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) cudaGetLastError();   // clusters of at most 8 then
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseSmem);
}

template <typename K>
static bool cluster_placeable(K* kernel, int ctas) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    int active = 0;
    coarse_config(ctas, kCoarseSmem, &cfg, at);
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&active, kernel, &cfg);
    if (e != cudaSuccess) cudaGetLastError();   // an unsupported size is not an error of the solve
    return e == cudaSuccess && active >= 1;
}

template <int DIM>
static cudaError_t coarse_attributes_all() {
    cudaError_t e = coarse_attributes(k_coarse<DIM, float, float>);
    if (e == cudaSuccess) e = coarse_attributes(k_coarse<DIM, __half, __half>);
    if (e == cudaSuccess) e = coarse_attributes(k_coarse<DIM, __nv_bfloat16, __nv_bfloat16>);
    if (e == cudaSuccess) e = coarse_attributes(k_adj_coarse<DIM>);
    return e;
}

template <int DIM>
static int largest_cluster() {
    for (int c = kMaxCtas; c > 1; c /= 2)
        if (cluster_placeable(k_coarse<DIM, float, float>, c) && cluster_placeable(k_coarse<DIM, __half, __half>, c) &&
            cluster_placeable(k_coarse<DIM, __nv_bfloat16, __nv_bfloat16>, c) && cluster_placeable(k_adj_coarse<DIM>, c))
            return c;
    return 1;
}

// Largest cluster this device places (16 is not a portable size), else one
// CTA; the first level that then runs in k_coarse.  Called outside any capture.
int coarse_setup(ss_sim* s) {
    // the attributes are the context's: for every simulation
    const cudaError_t e = s->dim == 3 ? coarse_attributes_all<3>() : coarse_attributes_all<2>();
    if (e != cudaSuccess) return check_cuda(e, "coarse cluster attributes");
    // the occupancy query takes milliseconds and its answer is the device's: once
    // per process and device
    static std::mutex mu;
    static std::map<int, int> known;   // 4 * device + dim -> CTAs
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lock(mu);
        int& c = known[4 * dev + s->dim];
        if (!c) c = s->dim == 3 ? largest_cluster<3>() : largest_cluster<2>();
        s->coarse_max_ctas = s->use_cluster ? c : 1;
    }
    s->coarse_from = s->levels;
    for (int l = s->levels - 1; l >= 1 && coarse_ctas(s, l, s->coarse_max_ctas); --l) s->coarse_from = l;
    return SS_OK;
}

// The arguments both kernels share; returns the cluster's CTAs (0: none fits) and
// its shared memory in floats.
template <int DIM, typename T>
static int coarse_args(const ss_sim* s, const ss_mg_schedule& mg, int L, T* const* p, T* const* r, CoarseArgs<T>& b,
                       long long* floats) {
    const int ctas = coarse_ctas(s, L, s->coarse_max_ctas);
    if (!ctas) return 0;
    b.nlev = s->levels - L;
    long long nw = 0, taps = 0;
    *floats = coarse_floats(s, L, ctas, &nw, &taps);
    int w = kZeros, tap = 0;
    for (int l = 0; l < b.nlev; ++l) {
        const ss::Level& lv = s->lv[L + l];
        for (int d = 0; d < 3; ++d) b.lv[l].n[d] = lv.n[d];
        b.lv[l].planes = level_planes(s, L + l, ctas, &b.lv[l].solo);
        b.lv[l].w = w;
        w += slab_floats<DIM>(lv.n, b.lv[l].planes);
        b.lv[l].tap = tap;
        tap += lv.n[0] + lv.n[1] + (DIM == 3 ? lv.n[2] : 0);
        b.lv[l].hh = lv.hh;
        b.lv[l].inv_hh = pow2_normal(lv.hh) ? 1.f / lv.hh : 0.f;
        b.p[l] = p[L + l];
        b.r[l] = r[L + l];
        b.alpha[l] = s->alpha[L + l];
    }
    b.nw = b.taps = (int)nw;
    b.fine = (int)(nw + 2 * taps);
    b.n_pre = mg.n_pre; b.n_post = mg.n_post; b.n_coarse = mg.n_coarse;
    return ctas;
}

template <int DIM, typename T>
static int launch_coarse_t(ss_sim* s, const ss_mg_schedule& mg, int L, T* const* p, T* const* r, bool p_zero, cudaStream_t st) {
    CoarseArgs<T> b{};
    long long floats = 0;
    const int ctas = coarse_args<DIM>(s, mg, L, p, r, b, &floats);
    if (!ctas) return set_error(SS_E_INVALID, "level too large for the coarse cluster");
    b.quirks = mg.ref_quirks ? 1 : 0;
    b.p_zero = p_zero ? 1 : 0;
    b.oob_smooth = smooth_oob(s, mg.ref_quirks);
    b.oob_resid = resid_oob(s, mg.ref_quirks);
    b.cmat = sizeof(T) == 2 ? s->cmat : nullptr;   // the mixed solve's coarse storage
    b.cpart = s->cmat_part;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    coarse_config(ctas, (size_t)floats * sizeof(float), &cfg, at);
    cfg.stream = st;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = s->pdl ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_coarse<DIM, T, T>, b);
    s->nlaunch += 1;
    return check_cuda(e, "k_coarse");
}

template <typename T>
static int launch_coarse_d(ss_sim* s, const ss_mg_schedule& mg, int L, T* const* p, T* const* r, bool p_zero, cudaStream_t st) {
    return s->dim == 3 ? launch_coarse_t<3, T>(s, mg, L, p, r, p_zero, st) : launch_coarse_t<2, T>(s, mg, L, p, r, p_zero, st);
}

int launch_coarse(ss_sim* s, const ss_mg_schedule& mg, int L, cudaStream_t st, bool p_zero) {
    return launch_coarse_d<float>(s, mg, L, s->p, s->r, p_zero, st);
}

int launch_coarse_mixed(ss_sim* s, const ss_mg_schedule& mg, int L, int prec, cudaStream_t st) {
    if (prec == SS_PREC_MIXED)
        return launch_coarse_d<__half>(s, mg, L, (__half* const*)s->cp, (__half* const*)s->cr, true, st);
    return launch_coarse_d<__nv_bfloat16>(s, mg, L, (__nv_bfloat16* const*)s->cp, (__nv_bfloat16* const*)s->cr, true, st);
}

// pbar, bbar: adjoint pressures and right-hand sides of all levels; the former's of
// level L is read, the latter's written.  cresp: the coarsest sweeps' response
// matrix (layout 0), or null; cpart: kProductLanes floats with it.
template <int DIM>
static int launch_adj_coarse_t(ss_sim* s, const ss_mg_schedule& mg, int L, const AdjScratch& w, cudaStream_t st) {
    CoarseArgs<float> b{};
    long long floats = 0;
    const int ctas = coarse_args<DIM>(s, mg, L, w.pbar, w.bbar, b, &floats);
    if (!ctas) return set_error(SS_E_INVALID, "level too large for the coarse cluster");
    b.oob_smooth = b.oob_resid = s->enclosed ? 1.f : 0.f;
    b.cmat = w.cresp;
    b.cpart = w.cpart;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    coarse_config(ctas, (size_t)floats * sizeof(float), &cfg, at);
    cfg.stream = st;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_adj_coarse<DIM>, b);
    s->nlaunch += 1;
    return check_cuda(e, "k_adj_coarse");
}

int launch_adj_coarse(ss_sim* s, const ss_mg_schedule& mg, int L, const AdjScratch& w, cudaStream_t st) {
    return s->dim == 3 ? launch_adj_coarse_t<3>(s, mg, L, w, st) : launch_adj_coarse_t<2>(s, mg, L, w, st);
}

// Response of the coarsest level's smoothing to unit right-hand sides: block
// i runs the `iters` red-black iterations from p = 0 with r = e_i (corrected
// out-of-grid rule, FP32 stores) and writes the result p as D[j * n + i] =
// dp_j / dr_i (layout 0: the adjoint applies D^T, reading consecutive i) or
// D[i * n + j] (layout 1: the mixed solve applies D, reading consecutive j).
// With `state`, blocks do nothing unless state[1] (set by k_coarse_check) asks
// for a rebuild.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_coarse_response(const __grid_constant__ CoarseArgs<float> b,
                                                              float* __restrict__ D, int layout,
                                                              const int* __restrict__ state) {
    if (state && state[1] == 0) return;
    float* F = smf();
    const Slab g = slab_of<DIM>(b, 0, 0);
    const int n = b.lv[0].n[0] * b.lv[0].n[1] * b.lv[0].n[2], i = blockIdx.x;
    for (int q = threadIdx.x; q < b.nw; q += kThreads) F[q] = 0.f;
    Cells<kCells> c;
    // the right-hand side is read from alpha's address space only to be replaced
    load_cells<DIM>(g, b.alpha[0], b.alpha[0], b.oob_smooth, b.oob_resid, c);
    int at[2][kCells];
#pragma unroll
    for (int j = 0; j < kCells; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            at[k][j] = -1;
            if (!c.in[k][j]) continue;
            at[k][j] = c.index(g, k, j);
            c.r[k][j] = at[k][j] == i ? 1.f : 0.f;
        }
    __syncthreads();
    solo_sweeps<DIM, float>(g, c, b.n_coarse);
#pragma unroll
    for (int j = 0; j < kCells; ++j)
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (at[k][j] >= 0)
                D[layout ? (size_t)i * n + at[k][j] : (size_t)at[k][j] * n + i] =
                    F[(k ? g.w[1] : g.w[0]) + threadIdx.x + j * kThreads];
}

// One block: state[1] = 1 when the coarsest level's solid fractions or the
// iteration count differ from the ones the matrix was built for (state[0];
// -1 before the first build), and the new ones are kept.
__global__ void __launch_bounds__(1024) k_coarse_check(const float* __restrict__ alpha, float* __restrict__ kept, int n,
                                                       int iters, int* __restrict__ state) {
    int diff = 0;
    for (int c = threadIdx.x; c < n; c += blockDim.x) diff |= alpha[c] != kept[c];
    diff = __syncthreads_or(diff) || state[0] != iters;
    for (int c = threadIdx.x; c < n; c += blockDim.x) kept[c] = alpha[c];
    if (threadIdx.x == 0) {
        state[0] = iters;
        state[1] = diff;
    }
}

static int launch_response(ss_sim* s, int iters, float* D, int layout, const int* state, cudaStream_t st) {
    const int l = s->levels - 1;
    const ss::Level& lv = s->lv[l];
    const int n = lv.n[0] * lv.n[1] * lv.n[2];
    CoarseArgs<float> b{};
    b.nlev = 1;
    for (int d = 0; d < 3; ++d) b.lv[0].n[d] = lv.n[d];
    b.lv[0].planes = level_planes(s, l, 1, &b.lv[0].solo);
    if (n > kCoarseResponseMax || !b.lv[0].planes)
        return set_error(SS_E_INVALID, "coarsest level too large for its response matrix");
    b.lv[0].hh = lv.hh;
    b.lv[0].w = kZeros;
    b.alpha[0] = s->alpha[l];
    b.nw = kZeros + (s->dim == 3 ? slab_floats<3>(lv.n, b.lv[0].planes) : slab_floats<2>(lv.n, b.lv[0].planes));
    b.n_coarse = iters;
    b.oob_smooth = b.oob_resid = smooth_oob(s, 0);
    const size_t smem = (size_t)b.nw * sizeof(float);
    auto kernel = s->dim == 3 ? k_coarse_response<3> : k_coarse_response<2>;
    kernel<<<n, kThreads, smem, st>>>(b, D, layout, state);
    s->nlaunch += 1;
    return check_cuda(cudaGetLastError(), "k_coarse_response");
}

int launch_coarse_response(ss_sim* s, int iters, float* D, cudaStream_t st) {
    return launch_response(s, iters, D, 0, nullptr, st);
}

// The mixed solve's coarsest-level matrix, rebuilt where the solid pyramid
// or the coarse iteration count changed since it was built.
int update_coarse_matrix(ss_sim* s, const ss_mg_schedule& mg, cudaStream_t st) {
    if (!s->cmat) return SS_OK;
    if (!s->cmat_dirty && s->cmat_iters == mg.n_coarse) return SS_OK;
    const ss::Level& lv = s->lv[s->levels - 1];
    const int n = lv.n[0] * lv.n[1] * lv.n[2];
    k_coarse_check<<<1, 1024, 0, st>>>(s->alpha[s->levels - 1], s->cmat_alpha, n, mg.n_coarse, s->cmat_state);
    s->nlaunch += 1;
    int rc = check_cuda(cudaGetLastError(), "k_coarse_check");
    if (rc == SS_OK) rc = launch_response(s, mg.n_coarse, s->cmat, 1, s->cmat_state, st);
    if (rc != SS_OK) return rc;
    s->cmat_dirty = 0;
    s->cmat_iters = mg.n_coarse;
    return SS_OK;
}

}  // namespace ss
