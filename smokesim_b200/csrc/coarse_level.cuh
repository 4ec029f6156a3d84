// coarse_level.cuh - per-cell multigrid operators of the per-level kernels
// (k_mg.cu), the out-of-grid rules and the coarsest level's matrix product, which
// the one-launch lower V-cycle (k_coarse.cu) uses too.  That one sums its cells from
// shared memory by code of its own, in the order of smooth_cell and residual_cell;
// the tests hold the two to the same bits.
#pragma once

#include "common.cuh"
#include "ss_internal.h"

namespace ss {

// T: storage type of p and r (float, or __half / __nv_bfloat16 on the coarse
// levels of the mixed-precision solve)
template <typename T>
struct MGArgsT {
    T* __restrict__ p;
    T* __restrict__ r;              // level right-hand side / residual (L >= 1)
    const float* __restrict__ alpha;  // L >= 1
    const uint8_t* __restrict__ flags;  // L == 0
    const float* __restrict__ div0;   // L == 0, smoother rule
    const float* __restrict__ div0r;  // L == 0, residual rule
    int nx, ny, nz;
    float oobA;     // solid fraction read for out-of-grid neighbours (0 = open, 1 = wall)
    float hh;       // h_L^2
    float rho_h;    // rho * h   (L == 0 smoother)
    float dt;
    float rho;
    float dt_h;     // dt * h    (L == 0 residual)
};
using MGArgs = MGArgsT<float>;

// Out-of-grid rule: ref_quirks keeps the reference's smoother (open, p = 0) /
// residual (wall) mismatch; the corrected mode uses the physical rule of the
// grid (wall when enclosed, open otherwise) in both operators.
static inline float smooth_oob(const ss_sim* s, int quirks) { return quirks ? 0.f : (s->enclosed ? 1.f : 0.f); }
static inline float resid_oob(const ss_sim* s, int quirks) { return quirks ? 1.f : (s->enclosed ? 1.f : 0.f); }

// ------------------------------------------------------------------ smoother
// smooth.comp:79-136 (2D :74-123): red-black Gauss-Seidel in place; solid
// cells and cells without fluid neighbours are skipped; out of grid = fluid
// with p = 0.
template <int DIM, bool L0, typename T = float>
SS_D void smooth_cell(const MGArgsT<T>& a, int x, int y, int z) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int c = idx3(x, y, z, nx, ny);
    float f_top, f_bottom, f_right, f_left, f_front = 0.f, f_back = 0.f;
    float r_c = 0.f;
    float p_top, p_bottom, p_right, p_left, p_front = 0.f, p_back = 0.f;
    auto load_p = [&]() {
        const T* P = a.p;
        p_top = y + 1 < ny ? ld(P[c + nx]) : 0.f;
        p_bottom = y > 0 ? ld(P[c - nx]) : 0.f;
        p_right = x + 1 < nx ? ld(P[c + 1]) : 0.f;
        p_left = x > 0 ? ld(P[c - 1]) : 0.f;
        if constexpr (DIM == 3) {
            p_front = z + 1 < nz ? ld(P[c + nx * ny]) : 0.f;
            p_back = z > 0 ? ld(P[c - nx * ny]) : 0.f;
        }
    };
    if constexpr (L0) {
        const uint8_t fl = a.flags[c];
        if (fl & F_SOLID) return;
        const float fo = 1.f - a.oobA;
        f_top = (fl & F_TOP) ? 0.f : (y + 1 < ny ? 1.f : fo);
        f_bottom = (fl & F_BOTTOM) ? 0.f : (y > 0 ? 1.f : fo);
        f_right = (fl & F_RIGHT) ? 0.f : (x + 1 < nx ? 1.f : fo);
        f_left = (fl & F_LEFT) ? 0.f : (x > 0 ? 1.f : fo);
        if constexpr (DIM == 3) {
            f_front = (fl & F_FRONT) ? 0.f : (z + 1 < nz ? 1.f : fo);
            f_back = (fl & F_BACK) ? 0.f : (z > 0 ? 1.f : fo);
        }
    } else {
        // every load of the cell is issued before the solid test, so one
        // memory latency covers the fraction, pressure and residual reads
        const float a_c = a.alpha[c];
        const float a_t = y + 1 < ny ? a.alpha[c + nx] : a.oobA;
        const float a_b = y > 0 ? a.alpha[c - nx] : a.oobA;
        const float a_r = x + 1 < nx ? a.alpha[c + 1] : a.oobA;
        const float a_l = x > 0 ? a.alpha[c - 1] : a.oobA;
        float a_f = 0.f, a_k = 0.f;
        if constexpr (DIM == 3) {
            a_f = z + 1 < nz ? a.alpha[c + nx * ny] : a.oobA;
            a_k = z > 0 ? a.alpha[c - nx * ny] : a.oobA;
        }
        r_c = ld(a.r[c]);
        load_p();
        if (a_c >= 1.f) return;
        f_top = 1.f - a_t;
        f_bottom = 1.f - a_b;
        f_right = 1.f - a_r;
        f_left = 1.f - a_l;
        if constexpr (DIM == 3) {
            f_front = 1.f - a_f;
            f_back = 1.f - a_k;
        }
    }
    if constexpr (L0) load_p();
    float f_sum = f_top + f_bottom + f_right + f_left;
    if constexpr (DIM == 3) f_sum = f_sum + f_front + f_back;
    if (f_sum == 0.f) return;
    float p_sum = p_top * f_top + p_bottom * f_bottom;
    p_sum = p_sum + p_right * f_right;
    p_sum = p_sum + p_left * f_left;
    if constexpr (DIM == 3) {
        p_sum = p_sum + p_front * f_front;
        p_sum = p_sum + p_back * f_back;
    }
    float pn;
    if constexpr (L0) pn = (p_sum - a.rho_h * a.div0[c] / a.dt) / f_sum;
    else pn = (p_sum - r_c * a.hh) / f_sum;
    a.p[c] = st<T>(pn);
}

// ------------------------------------------------------------------ residual
// compute_residual.comp:77-130 (2D :72-117): r = b - (sum_f p_nb - f_sum p)/h^2,
// out of grid = solid; level 0 takes b = rho*div/(dt*h).
template <int DIM, bool L0, typename T = float>
SS_D float residual_cell(const MGArgsT<T>& a, int x, int y, int z) {
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int c = idx3(x, y, z, nx, ny);
    float f_top, f_bottom, f_right, f_left, f_front = 0.f, f_back = 0.f;
    float p_top, p_bottom, p_right, p_left, p_front = 0.f, p_back = 0.f, p_c, old;
    const T* P = a.p;
    auto load_p = [&]() {
        p_top = y + 1 < ny ? ld(P[c + nx]) : 0.f;
        p_bottom = y > 0 ? ld(P[c - nx]) : 0.f;
        p_right = x + 1 < nx ? ld(P[c + 1]) : 0.f;
        p_left = x > 0 ? ld(P[c - 1]) : 0.f;
        if constexpr (DIM == 3) {
            p_front = z + 1 < nz ? ld(P[c + nx * ny]) : 0.f;
            p_back = z > 0 ? ld(P[c - nx * ny]) : 0.f;
        }
        p_c = ld(P[c]);
    };
    if constexpr (L0) {
        const uint8_t fl = a.flags[c];
        if (fl & F_SOLID) return 0.f;
        const float fo = 1.f - a.oobA;
        f_top = (fl & F_TOP) ? 0.f : (y + 1 < ny ? 1.f : fo);
        f_bottom = (fl & F_BOTTOM) ? 0.f : (y > 0 ? 1.f : fo);
        f_right = (fl & F_RIGHT) ? 0.f : (x + 1 < nx ? 1.f : fo);
        f_left = (fl & F_LEFT) ? 0.f : (x > 0 ? 1.f : fo);
        if constexpr (DIM == 3) {
            f_front = (fl & F_FRONT) ? 0.f : (z + 1 < nz ? 1.f : fo);
            f_back = (fl & F_BACK) ? 0.f : (z > 0 ? 1.f : fo);
        }
        load_p();
        old = a.rho * a.div0r[c] / a.dt_h;
    } else {
        // every load of the cell (fractions, pressures, right-hand side) is
        // issued before the solid test: one memory round trip a cell
        const float a_c = a.alpha[c];
        const float a_t = y + 1 < ny ? a.alpha[c + nx] : a.oobA;
        const float a_b = y > 0 ? a.alpha[c - nx] : a.oobA;
        const float a_r = x + 1 < nx ? a.alpha[c + 1] : a.oobA;
        const float a_l = x > 0 ? a.alpha[c - 1] : a.oobA;
        float a_f = 0.f, a_k = 0.f;
        if constexpr (DIM == 3) {
            a_f = z + 1 < nz ? a.alpha[c + nx * ny] : a.oobA;
            a_k = z > 0 ? a.alpha[c - nx * ny] : a.oobA;
        }
        load_p();
        old = ld(a.r[c]);
        if (a_c >= 1.f) return 0.f;
        f_top = 1.f - a_t;
        f_bottom = 1.f - a_b;
        f_right = 1.f - a_r;
        f_left = 1.f - a_l;
        if constexpr (DIM == 3) {
            f_front = 1.f - a_f;
            f_back = 1.f - a_k;
        }
    }
    float p_sum = p_top * f_top + p_bottom * f_bottom;
    p_sum = p_sum + p_right * f_right;
    p_sum = p_sum + p_left * f_left;
    float f_sum = f_top + f_bottom + f_right + f_left;
    if constexpr (DIM == 3) {
        p_sum = p_sum + p_front * f_front;
        p_sum = p_sum + p_back * f_back;
        f_sum = f_sum + f_front + f_back;
    }
    return old - (p_sum - f_sum * p_c) / a.hh;
}

// Part of p_j = sum_i E[i n + j] r_i over i in [i0, i1), where E[i n + j] =
// dp_j / dr_i of the coarsest level's n_coarse sweeps from p = 0
// (k_coarse_response, layout 1): eight partial sums taken round-robin
// ((i - i0) mod 8), added pairwise, so the oracle can repeat the order.  Two
// rounds of eight independent loads are in flight per step (the matrix
// streams from L2).
// r: the level's right-hand side, in shared memory.
SS_D float coarse_product(const float* __restrict__ E, const float* r, int n, int j, int i0, int i1) {
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const float* e = E + j;
    int i = i0;
    for (; i + 16 <= i1; i += 16) {
        float v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = __ldg(e + (size_t)(i + k) * n);
#pragma unroll
        for (int k = 0; k < 16; ++k) a[k & 7] += v[k] * r[i + k];
    }
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (i + k < i1) a[k & 7] += __ldg(e + (size_t)(i + k) * n) * r[i + k];
    return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// Slices of i per coarse value in the matrix product: the largest power of
// two (at most 32) with parts * n <= kProductLanes, twice the threads of the
// largest cluster - slices of at most 16 terms at 8^3.  The number depends on n
// alone, so every cluster size gives the same sums in the same order.
SS_D int coarse_parts(int n) {
    int parts = 1;
    while (parts < 32 && parts * 2 * n <= kProductLanes) parts *= 2;
    return parts;
}

// p_j = sum_i E[i n + j] r_i for every j of the coarsest level, in two phases
// separated by a barrier of the caller's.  Phase 1: item t is slice
// q = t / n of value j = t % n (adjacent lanes read adjacent j of a row of E,
// coalesced); its sum goes to part[q n + j].  Phase 2: value j folds its
// slices as a tree, v[q] += v[q + o] for o = parts/2 .. 1, rounds the result
// as R and stores it as PT.  `part` holds parts * n <= kProductLanes floats.
SS_D void coarse_matrix_partials(const float* __restrict__ E, const float* r, float* part, int n, int tid,
                                 int nthreads) {
    const int parts = coarse_parts(n), chunk = (n + parts - 1) / parts;
    for (int t = tid; t < parts * n; t += nthreads) {
        const int q = t / n, j = t % n;
        part[t] = coarse_product(E, r, n, j, q * chunk, min(n, (q + 1) * chunk));
    }
}

template <typename R, typename PT>
SS_D void coarse_matrix_fold(const float* part, PT* p, int n, int tid, int nthreads) {
    const int parts = coarse_parts(n);
    for (int j = tid; j < n; j += nthreads) {
        float v[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] = q < parts ? __ldcg(part + q * n + j) : 0.f;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1)
            if (o < parts) {
#pragma unroll
                for (int q = 0; q < o; ++q) v[q] = v[q] + v[q + o];
            }
        p[j] = st<PT>(rnd<R>(v[0]));
    }
}

}  // namespace ss
