// efl_vcycle.cuh — the lower levels of a multigrid V-cycle (multi_grid.rs:390-475) in one launch of one
// thread-block cluster.
//
// A V-cycle's coarse levels are a chain of dependent half-sweeps over few cells: launches (or one CTA's passes
// over L2) bound them, not arithmetic.  Here a cluster of 16 CTAs (8 where the device grants no more) holds every
// level of up to 256 x 256 cells in shared memory, in horizontal slabs of whole rows: the iterate with one halo
// row above and below, the right-hand side, the diagonal, the face fractions and one byte of flags per cell, all
// but the fractions per colour and compressed along x, so that a half-sweep reads consecutive words.  A
// half-sweep updates the slab's cells of one colour, stores the slab's edge rows into the neighbours' halo rows
// (distributed shared memory) and ends with the cluster's hardware barrier.  Slabs hold an even number of rows,
// so restriction and prolongation stay inside a slab; the smallest levels are gathered in the first CTA, where a
// block barrier is cheaper than the cluster's.  The coarse levels' geometry (restriction.wgsl:10-60 on the level
// set and the fractions) is restricted on the way, in shared memory.
//
// Same per-cell arithmetic and order of steps as the launch-per-step form (gs_update, residual_at, restrict_from,
// prolong_cell; smoother weight 1, resolution scale 2^level; symmetric: post-smoothing black then red), so the
// result is identical.  A cell whose four neighbours are fluid behind full faces ("standard": the fractions are 1
// and the diagonal is 4) skips the loads of its coefficients; 1 * x and x / 4 = x * 0.25 are exact.
//
// Latency bounds it: a half-sweep of a small level is one chain of dependent loads, sums and a division (250 cycles
// in f64, 275 in f32) and a barrier (the cluster's: 500 cycles).  So the coefficients sit in registers for a level's
// half-sweeps and the code of each step stands once.  Measured per call: 256^2 levels and below 74 us (f32) and 84
// (f64), 58 and 66 with the geometry kept; the one-CTA form took 120 us from 128^2 down, after 25 to 97 us for the
// 256^2 level's launches.
#pragma once

#include <cooperative_groups.h>
#include <cuda_pipeline.h>

#include <type_traits>

#include "efl_kernels.cuh"

namespace efl {

constexpr int VC_MAX_LEVELS = 14;
constexpr int VC_MAX_CELLS = 256 * 256;  // of the first level, if it fits the cluster's shared memory
enum { VC_GEOM_ONCE = 0, VC_GEOM_STORE = 1, VC_GEOM_LOAD = 2 };
constexpr int VC_THREADS = 512;
constexpr int VC_PAIRS = 4;  // pairs of cells a thread smooths at most (vc_plan)

// One level as the cluster holds it.  Offsets in bytes into every CTA's dynamic shared memory; per-colour arrays
// have rows of pitch HW = (nx + 1) / 2 + 2 entries, entry j + 1 is the cell x = 2 j + parity.
struct VcLevel {
    int nx, ny;
    int R;         // rows per slab (gathered: all)
    int hw, HW;
    int lc;        // threads: 2^lc columns (pairs of cells), 2^-lc of the block's threads rows
    int W;         // row pitch of the level set and the y fractions; the x fractions' is W + 2
    int ox, ob, oden, ofl, ols, ofu, ofv;
    int gathered;
};
template <class T>
struct VcArgs {
    VcLevel lv[VC_MAX_LEVELS];
    int count;      // levels
    int first;      // the first one's index in the whole V-cycle (resolution scale 2^first)
    int gather;     // the first gathered level (count: none)
    LevelT<T> top;  // level 0 here, in global memory
    int x_zero;     // its iterate starts at zero (not read)
    // The geometry (flags, diagonals, fractions, level sets of every level: bytes [oimg, oimg + nimg) of each CTA's
    // shared memory) does not change between the V-cycles of a solve: the first one stores it here (VC_GEOM_STORE)
    // and the others load it (VC_GEOM_LOAD) instead of restricting it again (80 -> 62 us a call in f32, 84 -> 66 in f64).
    unsigned char* image;
    int mode, oimg, nimg;
    T cdiv[VC_MAX_LEVELS], factor[VC_MAX_LEVELS];  // gs_cdiv, residual_factor per level
    int pre, post, coarsest, symmetric;
};

constexpr unsigned VC_UPDATE = 1, VC_FLUID = 2 /* 2, 4, 8, 16: left, right, up, down neighbour fluid */, VC_STD = 32,
                   VC_COUNTED = 64, VC_WET = 128 /* level set < 0 */;

template <class T>
__global__ void __launch_bounds__(VC_THREADS, 1) k_vcycle_cluster(const __grid_constant__ VcArgs<T> A) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(128) unsigned char sm[];
    constexpr int NT = VC_THREADS;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), tid = threadIdx.x;
    unsigned char* const up = cl.map_shared_rank(&sm[0], max(rank - 1, 0));
    unsigned char* const down = cl.map_shared_rank(&sm[0], min(rank + 1, (int)cl.num_blocks() - 1));
    unsigned char* const head = cl.map_shared_rank(&sm[0], 0);
    auto rows_from = [&](const VcLevel& V) { return V.gathered ? 0 : rank * V.R; };
    auto rows_of = [&](const VcLevel& V) {  // valid rows of this CTA's slab
        return V.gathered ? (rank == 0 ? V.ny : 0) : max(min(V.ny - rank * V.R, V.R), 0);
    };
    auto X = [&](unsigned char* s, const VcLevel& V, int c) { return reinterpret_cast<T*>(s + V.ox) + c * (V.R + 2) * V.HW; };
    auto B = [&](unsigned char* s, const VcLevel& V, int c) { return reinterpret_cast<T*>(s + V.ob) + c * V.R * V.HW; };
    auto DEN = [&](const VcLevel& V, int c) { return reinterpret_cast<T*>(sm + V.oden) + c * V.R * V.HW; };
    auto FL = [&](const VcLevel& V, int c) { return sm + V.ofl + c * V.R * V.HW; };
    auto LS = [&](unsigned char* s, const VcLevel& V) { return reinterpret_cast<float*>(s + V.ols); };  // [R + 2][W]
    auto FU = [&](unsigned char* s, const VcLevel& V) { return reinterpret_cast<float*>(s + V.ofu); };  // [R][W + 2]
    auto FV = [&](unsigned char* s, const VcLevel& V) { return reinterpret_cast<float*>(s + V.ofv); };  // [R + 1][W]
    // f(row, j) over rows x (pairs of columns) of a level: no divisions, a warp's threads side by side in x.
    auto each = [&](const VcLevel& V, int rows, auto f) {
        const int tx = tid & ((1 << V.lc) - 1), step = NT >> V.lc;
#pragma unroll 1
        for (int r = tid >> V.lc; r < rows; r += step)
#pragma unroll 1
            for (int j = tx; j < V.hw; j += 1 << V.lc) f(r, j);
    };

    // Flags and diagonals of the slab's cells (gs_update, residual_at).
    auto coefficients = [&](const VcLevel& V) {
        const int y0 = rows_from(V);
        const float *ls = LS(sm, V), *fu = FU(sm, V), *fv = FV(sm, V);
        each(V, rows_of(V), [&](int r, int j) {
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int x = 2 * j + o, y = y0 + r;
                if (x >= V.nx) continue;
                const float* l = ls + (r + 1) * V.W + x;
                const float phi = *l;
                const float f[4] = {fu[r * (V.W + 2) + x], fu[r * (V.W + 2) + x + 1], fv[r * V.W + x],
                                    fv[(r + 1) * V.W + x]};
                unsigned m = phi < 0.0f ? VC_WET : 0u;
                T den = T(0);
                if (!(phi >= 0.0f) && !(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
                    m |= VC_COUNTED;
                    const bool in[4] = {x > 0, x + 1 < V.nx, y > 0, y + 1 < V.ny};
                    const float nb[4] = {in[0] ? l[-1] : 0.0f, in[1] ? l[1] : 0.0f, in[2] ? l[-V.W] : 0.0f,
                                         in[3] ? l[V.W] : 0.0f};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (in[k]) {
                            if (nb[k] < 0.0f) {
                                den += (T)f[k];
                                m |= VC_FLUID << k;
                            } else {
                                den += (T)f[k] * (T(1) - (T)nb[k] / (T)phi);
                            }
                        }
                    if (!(fabs(den) < (T)1.0e-6f)) m |= VC_UPDATE;
                    if ((m & (15 * VC_FLUID)) == 15 * VC_FLUID && f[0] == 1.0f && f[1] == 1.0f && f[2] == 1.0f &&
                        f[3] == 1.0f)
                        m |= VC_STD;
                }
                const int c = (x + y) & 1, at = r * V.HW + j + 1;
                FL(V, c)[at] = (unsigned char)m;
                DEN(V, c)[at] = den;
            }
        });
    };
    // The coarse level C's level set and fractions from F's (restrict_from); edge rows into the neighbours' halos.
    auto restrict_geometry = [&](const VcLevel& F, const VcLevel& C) {
        const int fy0 = rows_from(F), fr = rows_of(F), cy0 = C.gathered && !F.gathered ? 0 : rows_from(C);
        const int Y0 = fy0 / 2, Y1 = min((fy0 + fr) / 2, C.ny);  // the coarse rows this slab's rows make
        unsigned char* to = C.gathered && !F.gathered ? head : sm;
        const float *ls = LS(sm, F), *fu = FU(sm, F), *fv = FV(sm, F);
        // a slab keeps the faces below its last row too (the row's y fractions only)
        const int rows = Y1 - Y0, extra = rows > 0 && (!C.gathered || Y1 == C.ny) ? 1 : 0;
        each(C, rows + extra, [&](int q, int j) {
            const int cr = Y0 + q - cy0, r = 2 * q;
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int x = 2 * j + o;
                if (x >= C.nx) continue;
                const float* g = fv + r * F.W + 2 * x;
                FV(to, C)[cr * C.W + x] = 0.5f * (g[0] + g[1]);
                if (q >= rows) continue;
                const float* l = ls + (r + 1) * F.W + 2 * x;
                const float ph0 = l[0], ph1 = l[F.W], ph2 = l[1], ph3 = l[F.W + 1];
                float pr = ph0;
                if (fabsf(ph1) < fabsf(pr)) pr = ph1;
                if (fabsf(ph2) < fabsf(pr)) pr = ph2;
                if (fabsf(ph3) < fabsf(pr)) pr = ph3;
                LS(to, C)[(cr + 1) * C.W + x] = pr;
                if (!C.gathered) {
                    if (cr == 0 && Y0 + q > 0) LS(up, C)[(C.R + 1) * C.W + x] = pr;
                    if (cr == C.R - 1 && Y0 + q + 1 < C.ny) LS(down, C)[x] = pr;
                }
                const float* f = fu + r * (F.W + 2) + 2 * x;
                FU(to, C)[cr * (C.W + 2) + x] = 0.5f * (f[0] + f[F.W + 2]);
                if (x == C.nx - 1) FU(to, C)[cr * (C.W + 2) + x + 1] = 0.5f * (f[2] + f[F.W + 4]);
            }
        });
    };
    // n red-black iterations (gs_update with weight 1), colour c0 first.  A thread keeps the coefficients of its NP
    // pairs of cells in registers for the call (weights 0 towards neighbours that are not fluid), so a half-sweep is
    // four loads, the update and a store.
    auto smooth_pairs = [&](auto np, const VcLevel& V, int n, int c0, T cdiv) {
        constexpr int NP = decltype(np)::value, G = NP < 2 ? NP : 2;
        const int y0 = rows_from(V), rows = rows_of(V), step = NT >> V.lc, ty = tid >> V.lc, j = tid & ((1 << V.lc) - 1);
        const int HW = V.HW, W = V.W;
        const bool col = j < V.hw;
        T cb[NP][2], dn[NP][2];
        float w[NP][2][4];
        unsigned upd = 0, general = 0;  // bit 2 p + s: update cell; a cell that is not standard in the warp
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int r = ty + p * step, at = r * HW + j + 1;
            const bool in = col && r < rows;
#pragma unroll
            for (int q = 0; q < 2; ++q) {  // q = 0: the colour that goes first
                const int c = q ? 1 - c0 : c0, x = 2 * j + ((y0 + r + c) & 1);
                const unsigned m = in ? FL(V, c)[at] : 0u;
                cb[p][q] = T(0);
                dn[p][q] = T(1);
#pragma unroll
                for (int k = 0; k < 4; ++k) w[p][q][k] = 0.0f;
                if (m & VC_UPDATE) {
                    const float *fu = FU(sm, V) + r * (W + 2) + x, *fv = FV(sm, V) + r * W + x;
                    const float f[4] = {fu[0], fu[1], fv[0], fv[W]};
#pragma unroll
                    for (int k = 0; k < 4; ++k) w[p][q][k] = m & (VC_FLUID << k) ? f[k] : 0.0f;
                    cb[p][q] = cdiv * B(sm, V, c)[at];
                    dn[p][q] = DEN(V, c)[at];
                    if constexpr (sizeof(T) == 8) dn[p][q] = T(1) / dn[p][q];
                    upd |= 1u << (2 * p + q);
                }
                // one path for a warp's G pairs
                if (__any_sync(0xffffffffu, (m & (VC_UPDATE | VC_STD)) == VC_UPDATE)) general |= 1u << (2 * (p / G * G) + q);
            }
        }
        // Everything that does not change between half-sweeps, so that one costs few instructions.
        const bool gathered = V.gathered;
        const int row = HW * (int)sizeof(T), plane = (V.R + 2) * row;
        int own[NP], side[NP][2];  // byte offsets: a pair's cells in colour plane c0; the word right of, per colour
        unsigned act = 0, push = 0;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const int r = ty + p * step;
            own[p] = V.ox + c0 * plane + (r + 1) * row + (j + 1) * (int)sizeof(T);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = q ? 1 - c0 : c0;
                side[p][q] = V.ox + (1 - c) * plane + (r + 1) * row + (j + 1 + ((y0 + r + c) & 1)) * (int)sizeof(T);
            }
            if (col && r < rows) act |= 1u << p;
            if (!gathered && r == 0 && y0 > 0) push |= 1u << p;
            if (!gathered && r == V.R - 1 && y0 + V.R < V.ny) push |= 16u << p;
        }
        const int flip = (1 - 2 * c0) * plane;  // from colour plane c0 to the other
        // halo rows in the neighbours: row R + 1 above, row 0 below
        unsigned char* const to_up = up + V.ox + c0 * plane + (V.R + 1) * row + (j + 1) * (int)sizeof(T);
        unsigned char* const to_down = down + V.ox + c0 * plane + (j + 1) * (int)sizeof(T);
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
                for (int p0 = 0; p0 < NP; p0 += G) {  // G pairs side by side
                    if (!(act & (1u << p0))) continue;  // a thread's later pairs lie further down
                    T* xc[G];
                    T xl[G], xr[G], xu[G], xd[G], old[G], pn[G];
#pragma unroll
                    for (int i = 0; i < G; ++i) {
                        const int p = p0 + i;
                        if (!(act & (1u << p))) {  // below the slab: the first pair's cells again, not stored
                            own[p] = own[p0];
                            side[p][q] = side[p0][q];
                        }
                        xc[i] = reinterpret_cast<T*>(sm + own[p] + (q ? flip : 0));
                        const unsigned char* const xo = sm + own[p] + (q ? 0 : flip);
                        const T* const o = reinterpret_cast<const T*>(sm + side[p][q]);
                        xl[i] = o[-1];
                        xr[i] = o[0];
                        xu[i] = *reinterpret_cast<const T*>(xo - row);
                        xd[i] = *reinterpret_cast<const T*>(xo + row);
                        old[i] = *xc[i];
                    }
                    if (general & (1u << (2 * p0 + q))) {
#pragma unroll
                        for (int i = 0; i < G; ++i) {
                            T nume = cb[p0 + i][q];
                            nume = nume + (T)w[p0 + i][q][0] * xl[i];
                            nume = nume + (T)w[p0 + i][q][1] * xr[i];
                            nume = nume + (T)w[p0 + i][q][2] * xu[i];
                            nume = nume + (T)w[p0 + i][q][3] * xd[i];
                            if constexpr (sizeof(T) == 8) pn[i] = nume * dn[p0 + i][q];
                            else pn[i] = (upd & (1u << (2 * (p0 + i) + q)) ? nume : T(1)) / dn[p0 + i][q];  // (0 / 1 is slow)
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < G; ++i) {
                            T nume = cb[p0 + i][q];
                            nume = nume + xl[i];
                            nume = nume + xr[i];
                            nume = nume + xu[i];
                            nume = nume + xd[i];
                            pn[i] = nume * T(0.25);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < G; ++i) {
                        const int p = p0 + i;
                        if (!(act & (1u << p))) continue;
                        const T v = upd & (1u << (2 * p + q)) ? T(1) * pn[i] + T(0) * old[i] : T(0);
                        *xc[i] = v;  // a column past an odd width holds a cell that nothing reads
                        if (push & (17u << p)) {
                            if (push & (1u << p)) *reinterpret_cast<T*>(to_up + (q ? flip : 0)) = v;
                            if (push & (16u << p)) *reinterpret_cast<T*>(to_down + (q ? flip : 0)) = v;
                        }
                    }
                }
                if (gathered) __syncthreads();
                else cl.sync();
            }
        }
    };
    auto smooth = [&](int l, int n, int c0) {
        const VcLevel& V = A.lv[l];
        const T cdiv = A.cdiv[l];
        if (V.R <= NT >> V.lc) smooth_pairs(std::integral_constant<int, 1>{}, V, n, c0, cdiv);
        else if (V.R <= 2 * (NT >> V.lc)) smooth_pairs(std::integral_constant<int, 2>{}, V, n, c0, cdiv);
        else smooth_pairs(std::integral_constant<int, VC_PAIRS>{}, V, n, c0, cdiv);
    };
    // residual_at of the slab's cell (x, row r)
    auto residual = [&](const VcLevel& V, T factor, int y0, int r, int x) -> T {
        const int y = y0 + r, c = (x + y) & 1, odd = x & 1, at = r * V.HW + (x >> 1) + 1, h = at + V.HW;
        const unsigned m = FL(V, c)[at];
        const T* xo = X(sm, V, 1 - c);
        const T xc = X(sm, V, c)[h], xl = xo[h - 1 + odd], xr = xo[h + odd], xu = xo[h - V.HW], xd = xo[h + V.HW];
        T res = B(sm, V, c)[at];
        const float *fu = FU(sm, V) + r * (V.W + 2) + x, *fv = FV(sm, V) + r * V.W + x;
        const T f[4] = {(T)fu[0], (T)fu[1], (T)fv[0], (T)fv[V.W]}, xn[4] = {xl, xr, xu, xd};
        if constexpr (sizeof(T) == 8) {
            T sum = T(0);
#pragma unroll
            for (int k = 0; k < 4; ++k) sum = m & (VC_FLUID << k) ? sum + f[k] * xn[k] : sum;
            res = res - factor * (DEN(V, c)[at] * xc - sum);
        } else {
            T t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = f[k] * (xc - xn[k]) * factor;
            const bool in[4] = {x > 0, x + 1 < V.nx, y > 0, y + 1 < V.ny};
            const int inb = (int)in[0] + (int)in[1] + (int)in[2] + (int)in[3];
            if (inb != __popc(m & (15 * VC_FLUID))) {  // a neighbour inside the domain that is not fluid
                const float* l = LS(sm, V) + (r + 1) * V.W + x;
                const float phi = *l;
                const int off[4] = {-1, 1, -V.W, V.W};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (in[k] && !(m & (VC_FLUID << k))) t[k] = f[k] * (T(1) - l[off[k]] / phi) * xc * factor;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) res = in[k] ? res - t[k] : res;
        }
        return m & VC_COUNTED ? res : T(0);
    };
    // The residual of F restricted to C's right-hand side.
    auto restrict_residual = [&](int l) {
        const VcLevel &F = A.lv[l], &C = A.lv[l + 1];
        const T factor = A.factor[l];
        const int fy0 = rows_from(F), fr = rows_of(F), cy0 = C.gathered && !F.gathered ? 0 : rows_from(C);
        const int Y0 = fy0 / 2, Y1 = min((fy0 + fr) / 2, C.ny);
        unsigned char* to = C.gathered && !F.gathered ? head : sm;
        // Two lanes per coarse cell, one per row of its children; the first adds them up.  The two have the same q and j,
        // so both come to each shuffle, which waits for them (the residuals branch per cell, and the other lanes of the
        // warp may have fewer rows).
        const int sub = tid & 1, j0 = (tid >> 1) & ((1 << F.lc) - 1), step = max((NT / 2) >> F.lc, 1);
        const int rows = Y1 - Y0, q0 = (tid >> 1) >> F.lc, jstep = min(1 << F.lc, NT / 2);
        const unsigned pair = 3u << (tid & 30);
#pragma unroll 1
        for (int q = q0; q < rows; q += step)
#pragma unroll 1
            for (int j = j0 & (jstep - 1); j < C.nx; j += jstep) {
                const T ra = residual(F, factor, fy0, 2 * q + sub, 2 * j);
                const T rb = residual(F, factor, fy0, 2 * q + sub, 2 * j + 1);
                const T ra1 = __shfl_xor_sync(pair, ra, 1), rb1 = __shfl_xor_sync(pair, rb, 1);
                if (sub == 0)
                    B(to, C, (j + Y0 + q) & 1)[(Y0 + q - cy0) * C.HW + (j >> 1) + 1] = T(0.25) * (ra + ra1 + rb + rb1);
            }
    };
    // prolong_cell: C's iterate added to F's where its level set is < 0; edge rows into the neighbours' halos.
    auto prolong = [&](int l) {
        const VcLevel &F = A.lv[l], &C = A.lv[l + 1];
        const int fy0 = rows_from(F), cy0 = C.gathered && !F.gathered ? 0 : rows_from(C);
        unsigned char* from = C.gathered && !F.gathered ? head : sm;
        const bool nb_up = !F.gathered && fy0 > 0, nb_down = !F.gathered && fy0 + F.R < F.ny;
        each(F, rows_of(F), [&](int r, int j) {  // the cells 2 j and 2 j + 1: coarse column j
            const int y = fy0 + r, cy = y >> 1, at = r * F.HW + j + 1;
            const bool in = j < C.nx && cy < C.ny;
            const T corr = in ? X(from, C, (j + cy) & 1)[(cy - cy0 + 1) * C.HW + (j >> 1) + 1] : T(0);
#pragma unroll
            for (int c = 0; c < 2; ++c) {  // one cell of each colour
                T* xf = X(sm, F, c) + at + F.HW;
                T v = *xf;
                if (in && (FL(F, c)[at] & VC_WET)) {
                    v = corr + v;
                    *xf = v;
                }
                if (r == 0 && nb_up) X(up, F, c)[(F.R + 1) * F.HW + j + 1] = v;
                if (r == F.R - 1 && nb_down) X(down, F, c)[j + 1] = v;
            }
        });
        if (F.gathered) __syncthreads();
        else cl.sync();
    };

    // ---- geometry
    const VcLevel& V0 = A.lv[0];
    const int y00 = rows_from(V0), rv0 = rows_of(V0);
    each(V0, rv0, [&](int r, int j) {  // the top level's right-hand side
        const int y = y00 + r, x = 2 * j;
        __pipeline_memcpy_async(&B(sm, V0, y & 1)[r * V0.HW + j + 1], &A.top.b.at(x, y), sizeof(T));
        __pipeline_memcpy_async(&B(sm, V0, (y & 1) ^ 1)[r * V0.HW + j + 1], &A.top.b.at(x + 1, y), sizeof(T));
    });
    __pipeline_commit();
    if (A.mode == VC_GEOM_LOAD) {
        const uint4* from = reinterpret_cast<const uint4*>(A.image + (size_t)rank * A.nimg);
        uint4* to = reinterpret_cast<uint4*>(sm + A.oimg);
        for (int i = tid; i < A.nimg / 16; i += NT) __pipeline_memcpy_async(&to[i], &from[i], 16);
        __pipeline_commit();
        __pipeline_wait_prior(0);
    } else {
#pragma unroll 1
        for (int l = 0; l < A.count; ++l) {  // flags 0: nothing is read past an odd width or a short slab
            const VcLevel& V = A.lv[l];
            unsigned* w = reinterpret_cast<unsigned*>(sm + V.ofl);  // padded to whole words
            for (int i = tid; i < (2 * V.R * V.HW + 3) / 4; i += NT) w[i] = 0u;
        }
        if (rv0 > 0)
            each(V0, rv0 + 2, [&](int q, int j) {  // rows -1 .. rv0; planes have a pitch of whole pairs and one more row
                const int r = q - 1, y = y00 + r, x = 2 * j;
                if (y >= 0 && y < V0.ny) __pipeline_memcpy_async(&LS(sm, V0)[q * V0.W + x], &A.top.ls.at(x, y), 8);
                if (r >= 0 && r <= rv0) __pipeline_memcpy_async(&FV(sm, V0)[r * V0.W + x], &A.top.fv.at(x, y), 8);
                if (r >= 0 && r < rv0) {
                    __pipeline_memcpy_async(&FU(sm, V0)[r * (V0.W + 2) + x], &A.top.fu.at(x, y), 8);
                    if (j == V0.hw - 1 && x + 2 == V0.nx)
                        __pipeline_memcpy_async(&FU(sm, V0)[r * (V0.W + 2) + x + 2], &A.top.fu.at(x + 2, y), 4);
                }
            });
        __pipeline_commit();
        __pipeline_wait_prior(0);
        cl.sync();  // every CTA of the cluster runs: its shared memory may be written from here on
#pragma unroll 1
        for (int l = 0; l < A.count; ++l) {
            const VcLevel& V = A.lv[l];
            if (V.gathered && rank != 0) break;
            coefficients(V);
            if (l + 1 == A.count) break;
            restrict_geometry(V, A.lv[l + 1]);
            if (V.gathered) __syncthreads();
            else cl.sync();
        }
        cl.sync();
        if (A.mode == VC_GEOM_STORE) {
            uint4* to = reinterpret_cast<uint4*>(A.image + (size_t)rank * A.nimg);
            const uint4* from = reinterpret_cast<const uint4*>(sm + A.oimg);
            for (int i = tid; i < A.nimg / 16; i += NT) to[i] = from[i];
        }
    }
    // ---- iterates: the top level's from memory (or zero), the others zero; halos and guards included
#pragma unroll 1
    for (int l = 0; l < A.count; ++l) {
        const VcLevel& V = A.lv[l];
        T* x = X(sm, V, 0);
        for (int i = tid; i < 2 * (V.R + 2) * V.HW; i += NT) x[i] = T(0);
    }
    if (!A.x_zero && rv0 > 0) {
        __syncthreads();
        each(V0, rv0 + 2, [&](int q, int j) {
            const int y = y00 + q - 1, x = 2 * j;
            if (y < 0 || y >= V0.ny) return;
            X(sm, V0, y & 1)[q * V0.HW + j + 1] = A.top.x.at(x, y);
            if (x + 1 < V0.nx) X(sm, V0, (y & 1) ^ 1)[q * V0.HW + j + 1] = A.top.x.at(x + 1, y);
        });
    }
    cl.sync();
    // ---- the V-cycle: down to the last level and up again (each step's code once: a few iterations a call, its
    // instruction fetches would otherwise take longer than its work)
    const int last = A.count - 1, g = A.gather;
#pragma unroll 1
    for (int i = 0; i <= 2 * last; ++i) {
        const bool down_leg = i < last, up_leg = i > last;
        const int l = up_leg ? 2 * last - i : i;
        if (l >= g && rank != 0) continue;  // the first CTA's levels
        if (up_leg) {
            if (l + 1 == g) cl.sync();  // the first CTA has finished them
            prolong(l);
        }
        smooth(l, i == last ? A.coarsest : down_leg ? A.pre : A.post, up_leg && A.symmetric ? 0 : 1);
        if (down_leg) {
            restrict_residual(l);
            if (l + 1 == g) cl.sync();
            else __syncthreads();
        }
    }
    if (g <= 0) cl.sync();
    each(V0, rv0, [&](int r, int j) {
        const int y = y00 + r, x = 2 * j;
        A.top.x.at(x, y) = X(sm, V0, y & 1)[(r + 1) * V0.HW + j + 1];
        if (x + 1 < V0.nx) A.top.x.at(x + 1, y) = X(sm, V0, (y & 1) ^ 1)[(r + 1) * V0.HW + j + 1];
    });
    cl.sync();  // no CTA leaves while its shared memory may still be accessed
}

// The cluster size this device grants k_vcycle_cluster<T> at the largest shared memory (0: no cluster fits).
template <class T>
inline int vc_cluster_size(size_t* smem_limit) {
    static int size[64] = {};  // 0 unknown, -1 none
    static size_t limit[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    if (!size[dev]) {
        int found = -1, optin = 0;
        const void* k = (const void*)k_vcycle_cluster<T>;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) == cudaSuccess &&
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
            for (int n : {16, 8}) {
                cudaLaunchConfig_t cfg = {};
                cudaLaunchAttribute at[1];
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim.x = n;
                at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
                cfg.gridDim = dim3(n);
                cfg.blockDim = dim3(VC_THREADS);
                cfg.dynamicSmemBytes = optin;
                cfg.attrs = at;
                cfg.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters >= 1) {
                    found = n;
                    break;
                }
            }
        cudaGetLastError();
        limit[dev] = (size_t)optin;
        size[dev] = found;
    }
    *smem_limit = limit[dev];
    return std::max(size[dev], 0);
}

// gs_cdiv and residual_factor of the levels, on the host (the same IEEE operations).
template <class T>
inline void vc_factors(VcArgs<T>* A, float dx, float rho, float dt) {
    for (int l = 0; l < A->count; ++l) {
        const T d = (T)((float)(1u << (A->first + l)) * dx);
        A->cdiv[l] = d * d * (T)rho / (T)dt;
        A->factor[l] = (T)dt / (T)rho / d / d;
    }
}

// The layout of levels mg[first ..] in a cluster of nc CTAs: true if it fits `limit` bytes per CTA.  Gathers the
// levels of at most 1024 cells in the first CTA (a block barrier is cheaper there than the cluster's), later
// levels only where that does not fit.
template <class T>
inline bool vc_plan(const std::vector<LevelT<T>>& mg, size_t first, int nc, size_t limit, VcArgs<T>* A, size_t* smem) {
    const int count = (int)(mg.size() - first);
    if (count > VC_MAX_LEVELS) return false;
    int g0 = 0;
    while (g0 < count && (int64_t)mg[first + g0].nx * mg[first + g0].ny > 1024) ++g0;
    for (int g = g0; g <= count; ++g) {
        // rows of a slab: even on every level that is restricted from a slab
        const int steps = g == count ? g - 1 : g;
        if (steps > 20) return false;
        const int unit = 1 << steps, ny = mg[first].ny;
        const int R0 = ((ny + nc - 1) / nc + unit - 1) / unit * unit;
        size_t off = 0;
        auto take = [&](size_t bytes) {
            const size_t at = off;
            off += (bytes + 15) / 16 * 16;
            return (int)at;
        };
        for (int l = 0; l < count; ++l) {
            const LevelT<T>& L = mg[first + l];
            VcLevel& V = A->lv[l];
            V.nx = L.nx;
            V.ny = L.ny;
            V.gathered = l >= g;
            V.R = V.gathered ? L.ny : R0 >> l;
            V.hw = (L.nx + 1) / 2;
            V.HW = V.hw + 2;
            V.W = 2 * V.hw;
            V.lc = 0;
            while ((1 << V.lc) < V.hw && (1 << V.lc) < VC_THREADS) ++V.lc;
            if ((1 << V.lc) < V.hw || V.R > VC_PAIRS * (VC_THREADS >> V.lc)) off = limit + 1;  // beyond smooth_pairs
            V.ox = take(2 * (size_t)(V.R + 2) * V.HW * sizeof(T));
            V.ob = take(2 * (size_t)V.R * V.HW * sizeof(T));
            if (off > limit) break;
        }
        A->oimg = (int)off;
        for (int l = 0; l < count && off <= limit; ++l) {
            VcLevel& V = A->lv[l];
            const size_t cells = 2 * (size_t)V.R * V.HW;
            V.oden = take(cells * sizeof(T));
            V.ofl = take((cells + 3) / 4 * 4);
            // the level set is needed after the set-up by the f32 residual only: f64 keeps it in the iterate's place
            V.ols = sizeof(T) == 8 ? V.ox : take((size_t)(V.R + 2) * V.W * 4);
            V.ofu = take((size_t)V.R * (V.W + 2) * 4);
            V.ofv = take((size_t)(V.R + 1) * V.W * 4);
        }
        A->nimg = (int)off - A->oimg;
        if (off <= limit) {
            A->count = count;
            A->first = (int)first;
            A->gather = g;
            A->top = mg[first];
            *smem = off;
            return true;
        }
    }
    return false;
}

}  // namespace efl
