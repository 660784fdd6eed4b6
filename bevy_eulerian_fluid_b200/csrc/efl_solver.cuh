// efl_solver.cuh — red-black Gauss-Seidel pressure solves
// (projection/shaders/gauss_seidel.wgsl:12-88, host loop gauss_seidel.rs:142-147).
//
// Forms:
//  * solve_gsmix_persistent: the tolerance-driven solve (mixed-precision
//    iterative refinement, below) as ONE cooperative launch over the tiles that
//    hold water.  Each CTA keeps its tile plus a halo of 2k cells on chip, so
//    that k red-black iterations run between two halo exchanges (temporal
//    blocking; the result is identical to k global sweeps because a half-sweep
//    only reads the other colour).  Halos are exchanged through L2 by words
//    that carry the number of their exchange, polled with a bound; the relative
//    residual is reduced the same way and tested on the device every
//    check_interval iterations, so the whole solve needs no host round trip.
//  * solve_gsmix_global: the same solve with global-memory kernels and a host
//    loop, for grids the persistent scheme does not cover.
//  * solve_gs32_persistent: fixed-count f32 sweeps as one cooperative launch,
//    for grids of at most one tile per SM.
//  * solve_gs32_tiled: fixed-count f32 sweeps through shared-memory tiles
//    (used when the TMA sweep of efl_sweep_tma.cuh is unavailable).
#pragma once

#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "efl_kernels.cuh"

namespace efl {

struct GridBarrier {
    unsigned int count;
    unsigned int gen;  // unused (layout kept)
    int error;  // the first wait that ran out: 1 a barrier, 2 an exchange (xch_poll)
    int pad;
};

struct SolveResult {
    unsigned int iterations;
    int converged;
    int error;  // 1: a wait of the first CTA ran out, 2: more tiles with water than CTAs
    int pad;
    double r0, r1;  // relative residual before / after
};
// Read back together: any CTA's wait may run out, after the last exchange too, when the first CTA, which writes the
// result, has what it waited for; only the barrier's flag says so then.
struct SolveState {
    SolveResult result;
    GridBarrier barrier;
};

struct SolverWorkspace {
    int nx = 0, ny = 0, device = 0;
    int num_sms = 0;
    SolveState* state = nullptr;    // device
    GridBarrier* barrier = nullptr;  // state's
    SolveResult* result = nullptr;   // state's
    SolveState* h_state = nullptr;  // pinned host
    double2* partials = nullptr;
    int max_blocks = 0;
    long long spin_limit = 0;  // grid-barrier polls before giving up (0: kBarrierSpinLimit)
    unsigned char* wet = nullptr;  // per 32 x 8 block: holds a cell with level set < 0 (k_wet_blocks)
    ulonglong2* xch = nullptr;     // the persistent solve's exchanges (its first solve allocates them)
    size_t xch_bytes = 0;
};


constexpr long long kBarrierSpinLimit = 1ll << 25;  // acquire polls (~ 1 s)

// Grid-wide barrier for a cooperative launch (all CTAs co-resident), with a
// bounded spin.  count only grows (it is zeroed before each launch): a CTA's
// acq_rel arrival returns its arrival number, arrivals of barrier e are
// numbers [e * nblocks, (e + 1) * nblocks) because no CTA reaches barrier
// e + 1 before all have arrived at e, so the CTA waits (acquire loads) until
// count reaches the end of its barrier's range; the last arriver leaves at
// once.  One atomic round trip on the way in, none on the way out.  A CTA
// that polls `limit` times (kBarrierSpinLimit unless the caller set a
// shorter limit) sets barrier->error and leaves; the others see the flag
// while they wait (checked every 1024 polls) and leave too.
EFL_DEV bool grid_barrier(GridBarrier* gb, unsigned nblocks, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned arrived, cur;
        asm volatile("atom.acq_rel.gpu.add.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(&gb->count) : "memory");
        const unsigned target = (arrived / nblocks + 1) * nblocks;
        if (arrived + 1 != target) {
            long long spins = 0;
            for (;;) {
                asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(cur) : "l"(&gb->count) : "memory");
                if ((int)(cur - target) >= 0) break;
                if ((++spins & 1023) == 0 || spins >= limit) {
                    int e;
                    asm volatile("ld.acquire.gpu.s32 %0, [%1];" : "=r"(e) : "l"(&gb->error) : "memory");
                    if (e || spins >= limit) {
                        atomicExch(&gb->error, 1);
                        ok = 0;
                        break;
                    }
                }
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

struct PersistentParams {
    Level64 L;  // level 0: x = FP64 iterate (global), b = widened divergence
    int tiles_x;
    double cdiv;    // ((dx*dx)*rho)/dt (gauss_seidel.wgsl:58)
    double factor;  // dt/rho/dx/dx (residual.wgsl:34)
    double weight;
    double tol;
    unsigned max_iters, check_interval;
    double2* partials;
    GridBarrier* barrier;
    SolveResult* result;
    long long spin_limit;  // grid-barrier polls before giving up
    ulonglong2* xch;       // the exchanges' tagged words (oct_xch_bytes)
    float one;             // 1.0f, passed at run time (see x2_add1)
    const unsigned char* wet;  // per 32 x 8 block of cells (row pitch wet_w): holds a cell with level set < 0
    int wet_w, ntiles;
    int retry;             // run only if the launch before this one found too many tiles (result->error == 2)
};

constexpr unsigned char MODE_SKIP = 0;     // outside the domain or on the tile's outer ring
constexpr unsigned char MODE_ZERO = 1;     // air, fully solid or |denom| < 1e-6: p = 0
constexpr unsigned char MODE_UPDATE = 2;   // regular update
constexpr unsigned char MODE_COUNTED = 4;  // counted in the residual norms
constexpr unsigned char MODE_STD = 8;      // update cell with w = (1, 1, 1, 1), inv = 0.25 (coefficients implied)

// Sum of all CTAs' partials in CTA order; identical in every CTA.
EFL_DEV double ps_total_relative(const double2* partials, int nblocks) {
    // Warp 0: lane l adds partials l, l + 32, ... in order (independent loads,
    // one round of latency), then a fixed xor-shuffle tree; the same in every CTA.
    __shared__ double s_rel;
    if (threadIdx.x < 32) {
        double r = 0.0, b = 0.0;
        int i = threadIdx.x;
        for (; i + 96 < nblocks; i += 128) {  // four loads in flight, added in the same order
            const double2 v0 = __ldcg(&partials[i]), v1 = __ldcg(&partials[i + 32]);
            const double2 v2 = __ldcg(&partials[i + 64]), v3 = __ldcg(&partials[i + 96]);
            r += v0.x;
            b += v0.y;
            r += v1.x;
            b += v1.y;
            r += v2.x;
            b += v2.y;
            r += v3.x;
            b += v3.y;
        }
        for (; i < nblocks; i += 32) {
            const double2 v = __ldcg(&partials[i]);
            r += v.x;
            b += v.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            r += __shfl_xor_sync(0xffffffffu, r, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (threadIdx.x == 0)
            s_rel = b > 0.0 ? sqrt(r) / sqrt(b) : (r > 0.0 ? __longlong_as_double(0x7ff0000000000000ll) : 0.0);
    }
    __syncthreads();
    double v = s_rel;
    __syncthreads();
    return v;
}

inline efl_status solver_init(SolverWorkspace& ws, int nx, int ny, int device, std::string* err) {
    ws.nx = nx;
    ws.ny = ny;
    ws.device = device;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) {
        *err = "cudaGetDeviceProperties failed";
        return EFL_ERR_CUDA;
    }
    ws.num_sms = prop.multiProcessorCount;
    ws.max_blocks = 4 * ws.num_sms;
    if (cudaMalloc(&ws.state, sizeof(SolveState)) != cudaSuccess ||
        cudaMalloc(&ws.partials, ws.max_blocks * sizeof(double2)) != cudaSuccess ||
        cudaMalloc(&ws.wet, (size_t)((nx + 31) / 32) * ((ny + 7) / 8)) != cudaSuccess ||
        cudaMallocHost(&ws.h_state, sizeof(SolveState)) != cudaSuccess) {
        *err = "solver workspace allocation failed";
        return EFL_ERR_OUT_OF_MEMORY;
    }
    ws.barrier = &ws.state->barrier;
    ws.result = &ws.state->result;
    return EFL_OK;
}
inline void solver_free(SolverWorkspace& ws) {
    if (ws.state) cudaFree(ws.state);
    if (ws.partials) cudaFree(ws.partials);
    if (ws.xch) cudaFree(ws.xch);
    if (ws.wet) cudaFree(ws.wet);
    if (ws.h_state) cudaFreeHost(ws.h_state);
    ws = SolverWorkspace{};
}

// ---------------------------------------------------------------------------
// Tolerance-driven solve in mixed-precision iterative-refinement form.
// Every check block of n iterations: the FP64 residual r of the FP64 iterate
// p (operator of residual.wgsl in factored form) gives the convergence test
// and the f32 right-hand side rc = f32(cdiv * r); n SOR red-black
// iterations then run in f32 on the correction d (starting at 0) with f32
// coefficients w_k (face fraction of fluid in-bounds neighbours, else 0) and
// inv = f32(1/denom); then p += d in FP64, and the cells the reference sets
// to zero (air, fully solid, |denom| < 1e-6) get p = 0.  SOR is affine, so
// in exact arithmetic these are the RBGS iterates themselves: the
// iteration counts are those of red-black Gauss-Seidel, while the sweeps move
// f32 data.
// ---------------------------------------------------------------------------
// Paired-lane form of the persistent mixed solve (4 x 2 cells per thread).
//
// One cooperative launch = one solve (the f32 update in the same
// operation order on every cell, the same FP64 checks), with each thread
// owning a 4 x 2 block of the extended tile: cells c0..c3 in its upper row,
// c4..c7 in its lower one.  A half-sweep updates four of them, in two pairs
// of one colour (c0, c2) and (c5, c7), or (c1, c3) and (c4, c6), and the two
// cells of a pair are the two lanes of Blackwell's paired f32 instructions
// (mul.rn.f32x2 for the products, fma.rn.f32x2 by a run-time 1.0 for the
// sums: per lane the IEEE-rounded f32 product and sum, so each lane is the
// scalar update exactly).  The layout makes the operand pairs fall out of it:
//  * in the colour-compressed shared image of the correction
//    (d[k][y][x / 2]) a pair's two cells are adjacent words, so one 8-byte
//    load brings both neighbours above (or below) a pair and one 8-byte store
//    publishes the pair;
//  * of the eight neighbour values a pair needs, four come from the thread's
//    own registers as ready-made pairs, two from one 8-byte load and two
//    (left of c0 / c4, right of c3 / c7) from a 4-byte load packed with a
//    register lane;
//  * the face weights, 1/den and the right-hand side stay in registers as
//    lane pairs for the whole solve.
// Cells on the tile image's outermost ring update too, from clamped
// neighbour values: their results are as wrong as the stale values a frozen
// ring would hold, and like those they move inwards one ring per half-sweep,
// so the owned cells are exact after the 2K half-sweeps between exchanges
// (every value stays finite, and the exchange reloads the ring).
typedef unsigned long long f32x2;  // lane 0 = low word
EFL_DEV f32x2 x2_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
EFL_DEV float x2_lane(f32x2 v, int lane) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return lane ? b : a;
}
EFL_DEV f32x2 x2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// round(a + c) per lane, written as fma(a, one, c) with one = 1.0 known only at
// run time.  ptxas contracts a paired product feeding a paired add (mul.rn /
// add.rn f32x2) into one fused multiply-add, -fmad=false notwithstanding,
// which drops the product's rounding; a product feeding the multiplicand of
// an FMA by an unknown factor cannot be contracted, and a * 1 + c rounds once,
// exactly like the add (signed zeros included).
EFL_DEV f32x2 x2_add1(f32x2 a, f32x2 one, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(one), "l"(c));
    return r;
}
// The update of two cells: nume = rc + wl L + wr R + wu U + wd D (in that
// order, each product rounded), d' = wgt (nume inv) + omw d.
EFL_DEV f32x2 oct_update(f32x2 rc, f32x2 wl, f32x2 wr, f32x2 wu, f32x2 wd, f32x2 inv, f32x2 omw, f32x2 d, f32x2 L,
                         f32x2 R, f32x2 U, f32x2 D, f32x2 wgt, f32x2 one) {
    f32x2 n = x2_add1(x2_mul(wl, L), one, rc);
    n = x2_add1(x2_mul(wr, R), one, n);
    n = x2_add1(x2_mul(wu, U), one, n);
    n = x2_add1(x2_mul(wd, D), one, n);
    return x2_add1(x2_mul(wgt, x2_mul(n, inv)), one, x2_mul(omw, d));
}

template <int EX, int EY, int ROWS>
struct OctTile {
    static constexpr int W2 = EX / 2, W4 = EX / 4, NB = (EX / 4) * (EY / ROWS);
    static constexpr int WP = W2 % 16 == 4 ? W2 : W2 + ((4 - W2 % 16) + 16) % 16;  // row stride of d (words)
    // The FP64 planes hold cell (x, y) at y * RS + (x & 3) * W4 + (x >> 2): the threads of a warp (consecutive
    // blocks) reading the same cell of their blocks read consecutive words, and RS puts the next row of
    // blocks (ROWS rows down) 16 banks over, so a half-warp that spans two block rows does not conflict.
    static constexpr int rs_pad() {
        int pad = 0;
        while ((ROWS * (4 * W4 + pad)) % 16 != 8 && pad < 16) ++pad;
        return pad;
    }
    static constexpr int RS = 4 * W4 + rs_pad();
    EFL_DEV static int ix(int y, int x) { return y * RS + (x & 3) * W4 + (x >> 2); }
    double p[EY * RS];
    double b[EY * RS];
    double den[EY * RS];
    float d[2][EY][WP];  // [k][y][x / 2], k = (x + y) & 1 in the image (k = 0: the tile's base colour)
};

// Cell q of a thread's 4 x ROWS block sits at (i, j) = (q & 3, q >> 2); its colour in the image is
// k = (i + j) & 1, and it is lane i >> 1 of pair 2 j + k: the pair of the two cells of colour k in row j,
// which are adjacent words (2 bx, 2 bx + 1) of the colour-compressed image.
EFL_DEV constexpr int oct_pair(int q) { return 2 * (q >> 2) + (((q & 3) + (q >> 2)) & 1); }
EFL_DEV constexpr int oct_lane(int q) { return (q & 3) >> 1; }

// Exchanges between the CTAs of a solve: words of 32 bits of data under a 32-bit tag, written and polled as 64-bit
// relaxed accesses, which are indivisible.  The receiver waits for the tag of the exchange on the data itself, so an
// exchange costs a store and a load of L2 and no fence, no flag and no barrier (a grid barrier and the loads behind it
// took 3 us of every 8 iterations: 0.94 us per iteration on a 512^2 pool; 0.69 now, 0.38 of them half-sweeps).  Tags only
// grow within a solve and the words are cleared before its first barrier; two buffers alternate, which suffices because
// every CTA waits in each exchange for all the CTAs that read its words.
EFL_DEV void xch_store(ulonglong2* p, uint32_t a, uint32_t b, uint32_t tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | a), "l"(t | b) : "memory");
}
// N pairs of words `stride` apart, when all carry the tag.  False: `limit` polls, or another CTA's, ran out.
template <int N>
EFL_DEV bool xch_poll(const ulonglong2* p, int stride, uint32_t tag, ulonglong2 (&w)[N], GridBarrier* gb,
                      long long limit) {
    for (long long spins = 0;;) {
#pragma unroll
        for (int k = 0; k < N; ++k)
            asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                         : "=l"(w[k].x), "=l"(w[k].y)
                         : "l"(p + (size_t)k * stride)
                         : "memory");
        bool got = true;
#pragma unroll
        for (int k = 0; k < N; ++k) got = got && (uint32_t)(w[k].x >> 32) == tag && (uint32_t)(w[k].y >> 32) == tag;
        if (got) return true;
        if ((++spins & 1023) == 0 || spins >= limit) {
            int e;
            asm volatile("ld.acquire.gpu.s32 %0, [%1];" : "=r"(e) : "l"(&gb->error) : "memory");
            if (e || spins >= limit) {
                atomicCAS(&gb->error, 0, 2);
                return false;
            }
        }
    }
}
EFL_DEV double xch_double(ulonglong2 w) {
    return __longlong_as_double((long long)((w.x & 0xffffffffull) | (w.y << 32)));
}
EFL_DEV void xch_store(ulonglong2* p, double v, uint32_t tag) {
    xch_store(p, (uint32_t)__double2loint(v), (uint32_t)__double2hiint(v), tag);
}

// The tiles (TX x TY owned cells, multiples of 32 and 8) of a level that hold a cell with level set < 0, in tile order,
// and after them the others: list[0 .. *n), list[*n .. ntiles).  The whole CTA calls it.
constexpr int OCT_MAX_TILES = 1024;
constexpr size_t OCT_XCH_SUMS = 2 * 2 * OCT_MAX_TILES;  // the residual sums of every CTA, then its cells
// Bytes of the exchanges of `ctas` CTAs that own `cells` cells each.
inline size_t oct_xch_bytes(int ctas, int cells) { return (OCT_XCH_SUMS + (size_t)ctas * cells) * sizeof(ulonglong2); }
constexpr int OCT_MAX_CTAS = 512;  // of one solve
// The sums of check `tag`: fetched by the CTA's first threads, ...
template <int NT>
EFL_DEV bool oct_fetch_sums(const ulonglong2* sums, uint32_t tag, int nblocks, GridBarrier* gb, long long limit,
                            double2* s_sums) {
    bool got = true;
    for (int i = threadIdx.x; i < nblocks; i += NT) {
        ulonglong2 w[2];
        got = xch_poll(sums + ((tag & 1) * OCT_MAX_TILES + i) * 2, 1, tag, w, gb, limit) && got;
        s_sums[i] = make_double2(xch_double(w[0]), xch_double(w[1]));
    }
    return got;
}
// ... and after a barrier added by every warp, in ps_total_relative's order.
EFL_DEV double oct_total_relative(const double2* s_sums, int nblocks) {
    double r = 0.0, b = 0.0;
    for (int i = threadIdx.x & 31; i < nblocks; i += 32) {
        r += s_sums[i].x;
        b += s_sums[i].y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        r += __shfl_xor_sync(0xffffffffu, r, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    return b > 0.0 ? sqrt(r) / sqrt(b) : (r > 0.0 ? __longlong_as_double(0x7ff0000000000000ll) : 0.0);
}
// The smallest tiles first: a CTA's sweeps cover its image, 64 x 64 cells here, and tiles without water need no CTA, so
// 32 x 32 tiles fit the device up to 148 x 1024 cells of water.  0.69 us per red-black iteration on a 512^2 pool.
// Before the checks shared its last exchange, 0.74; then the same tile by 4 x 2 blocks of cells (512 threads) took 0.79,
// exchanged every 6 iterations 0.86, every 4 iterations 0.91 (0.80 by 4 x 2 blocks), every 2 iterations 1.20.
#define OCT_SMALL 64, 64, 8, 256, 4
// Twice the cells per CTA, by 4 x 2 blocks so that a thread's coefficients stay in its registers: 0.90 us on a full
// 768 x 640 pool; by 4 x 4 blocks 1.00 (256 threads) against 0.93 then, exchanged every 8 iterations 1.40 (spilled).
#define OCT_MEDIUM 80, 48, 4, 480, 2
template <int TX, int TY, int NT>
EFL_DEV void oct_tiles(const PersistentParams& P, unsigned short* list, int* n) {
    static_assert(TX % 32 == 0 && TY % 8 == 0, "whole blocks");
    __shared__ unsigned char hot[OCT_MAX_TILES];
    const int wet_h = (P.L.ny + 7) / 8;
    for (int t = threadIdx.x; t < P.ntiles; t += NT) {
        const int bx = (t % P.tiles_x) * (TX / 32), by = (t / P.tiles_x) * (TY / 8);
        unsigned any = 0;
#pragma unroll
        for (int j = 0; j < TY / 8; ++j)
#pragma unroll
            for (int i = 0; i < TX / 32; ++i)
                any |= bx + i < P.wet_w && by + j < wet_h ? P.wet[(by + j) * P.wet_w + bx + i] : 0u;
        hot[t] = any != 0;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int total = 0, at = 0;
        for (int t0 = 0; t0 < P.ntiles; t0 += 32)
            total += __popc(__ballot_sync(0xffffffffu, t0 + lane < P.ntiles && hot[t0 + lane]));
        int cold = total;
        for (int t0 = 0; t0 < P.ntiles; t0 += 32) {
            const bool in = t0 + lane < P.ntiles, h = in && hot[t0 + lane];
            const unsigned mh = __ballot_sync(0xffffffffu, h), mc = __ballot_sync(0xffffffffu, in && !h);
            const unsigned below = (1u << lane) - 1u;
            if (h) list[at + __popc(mh & below)] = (unsigned short)(t0 + lane);
            else if (in) list[cold + __popc(mc & below)] = (unsigned short)(t0 + lane);
            at += __popc(mh);
            cold += __popc(mc);
        }
        if (lane == 0) *n = total;
    }
    __syncthreads();
}

// One simulation's solve by `nblocks` CTAs, this one being number `rank` of them and owning tile list[rank] (the
// simulation's active tiles: a tile without a cell of level set < 0 takes no part, as its correction is 0 and no
// weight points at its cells).  beat(rank) at each check, from the CTA's first thread.  False: a wait ran out.
struct OctNoBeat {
    EFL_DEV void operator()(unsigned) const {}
};
template <int EX, int EY, int KMAX, int NT, int ROWS, class Beat = OctNoBeat>
EFL_DEV bool oct_solve(const PersistentParams& P, const unsigned short* list, unsigned rank, unsigned nblocks,
                       Beat beat = Beat()) {
    using Tile = OctTile<EX, EY, ROWS>;
    constexpr int NC = 4 * ROWS, NPAIR = 2 * ROWS;
    static_assert(KMAX >= 1 && EX % 4 == 0 && EY % ROWS == 0 && ROWS % 2 == 0, "4 x ROWS blocks");
    static_assert(Tile::NB <= NT && NT % 32 == 0, "one thread per block");
    static_assert((2 * KMAX) % 4 == 0 && (2 * KMAX) % ROWS == 0, "halo of whole blocks");
    static_assert(NC <= 16, "cell flags in 64 bits");
    extern __shared__ __align__(16) unsigned char ps_raw[];
    Tile& T = *reinterpret_cast<Tile*>(ps_raw);
    constexpr int H = 2 * KMAX, W2 = Tile::W2, W4 = Tile::W4, NB = Tile::NB, WP = Tile::WP;
    constexpr int TXo = EX - 2 * H, TYo = EY - 2 * H;
    const Level64& L = P.L;
    const int tile = list[rank];
    const int gx0 = (tile % P.tiles_x) * TXo - H, gy0 = (tile / P.tiles_x) * TYo - H;
    const bool active = threadIdx.x < NB;
    const int bx = active ? (int)threadIdx.x % W4 : 0, by = active ? (int)threadIdx.x / W4 : 0;
    const int base = (gx0 + gy0) & 1;  // colour of the k = 0 cells (1 = red, (x + y) odd)
    const bool owned = active && bx >= H / 4 && bx < (H + TXo) / 4 && by >= H / ROWS && by < (H + TYo) / ROWS;
    const int x0 = 4 * bx, y0 = ROWS * by;
    // The words of this thread's block in its owner's part of an exchange: pair pi of corrections at [pi][block].
    // Null: the block is outside the domain, or its tile takes no part.
    constexpr int NBLK = (TXo / 4) * (TYo / ROWS), XP = NPAIR * NBLK;
    ulonglong2* part_of = nullptr;
    {
        const int gx = gx0 + x0, gy = gy0 + y0;
        const int tx = gx / TXo, ty = gy / TYo, t = ty * P.tiles_x + tx;
        if (active && gx >= 0 && gy >= 0 && tx < P.tiles_x && t < P.ntiles) {
            int lo = 0, hi = (int)nblocks;  // the tile's place among the first nblocks of the list (ascending)
            while (lo < hi) {
                const int m = (lo + hi) / 2;
                if (list[m] < t) lo = m + 1;
                else hi = m;
            }
            if (lo < (int)nblocks && list[lo] == t)
                part_of = P.xch + OCT_XCH_SUMS + (size_t)lo * (2 * XP) + (gy - ty * TYo) / ROWS * (TXo / 4) + (gx - tx * TXo) / 4;
        }
    }
    for (int i = threadIdx.x; i < 2 * XP; i += NT) P.xch[OCT_XCH_SUMS + (size_t)rank * (2 * XP) + i] = make_ulonglong2(0, 0);
    if (threadIdx.x < 4) P.xch[((threadIdx.x >> 1) * OCT_MAX_TILES + rank) * 2 + (threadIdx.x & 1)] = make_ulonglong2(0, 0);
    // FP64 plane index of the cell (x0 + i, y0 + j), i in -1 .. 4 and j in -1 .. ROWS (constants once unrolled)
    const int pbase = y0 * Tile::RS + bx;
    auto pix = [&](int i, int j) { return pbase + j * Tile::RS + (i & 3) * W4 + (i >> 2); };
    const float wgt = (float)P.weight, omw1 = 1.0f - (float)P.weight;
    // bit q: update cell, live (not on the image's outermost ring); 32 + q: counted and live; 48 + q: owned and in the
    // domain.  Bits 16 + q, live, are not read: without them the 80 x 72 image's form spills 796 bytes, not 612.
    unsigned long long fl = 0;
    unsigned upd_halo = 0;  // bit q: update cell, the image's outermost ring included
    f32x2 wl[NPAIR], wr[NPAIR], wu[NPAIR], wd[NPAIR], inv[NPAIR], rc[NPAIR], dv[NPAIR];
    {
        float fw[4][NC], finv[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            const int lx = x0 + (q & 3), ly = y0 + (q >> 2);
            const int gx = gx0 + lx, gy = gy0 + ly;
            const bool live = active && lx > 0 && lx < EX - 1 && ly > 0 && ly < EY - 1;
            if (live) fl |= 1ull << (16 + q);
            float wv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            finv[q] = 0.0f;
            double den = 0.0, bb = 0.0, pv = 0.0;
            if (active && (unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny) {
                const float phi = L.ls.at(gx, gy);
                bb = L.b.at(gx, gy);
                pv = __ldcg(&L.x.p[(size_t)gy * L.x.P + gx]);
                if (owned) fl |= 1ull << (48 + q);
                if (phi < 0.0f) {
                    const float f[4] = {L.fu.at(gx, gy), L.fu.at(gx + 1, gy), L.fv.at(gx, gy), L.fv.at(gx, gy + 1)};
                    if (!(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
                        if (live) fl |= 1ull << (32 + q);
                        const int ox[4] = {-1, 1, 0, 0}, oy[4] = {0, 0, -1, 1};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int jx = gx + ox[k], jy = gy + oy[k];
                            if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
                                const float level = L.ls.at(jx, jy);
                                if (level < 0.0f) {
                                    den += (double)f[k];
                                    wv[k] = f[k];
                                } else {
                                    den += (double)f[k] * (1.0 - (double)level / (double)phi);
                                }
                            }
                        }
                        if (!(fabs(den) < (double)1.0e-6f)) {
                            if (live) fl |= 1ull << q;
                            upd_halo |= 1u << q;
                            finv[q] = (float)(1.0 / den);
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) fw[k][q] = wv[k];
            if (active) {
                T.p[pix(q & 3, q >> 2)] = pv;
                T.b[pix(q & 3, q >> 2)] = bb;
                T.den[pix(q & 3, q >> 2)] = den;
            }
        }
        // pair 2 j + k = the cells (i0, j), (i0 + 2, j) with i0 = (k + j) & 1
#pragma unroll
        for (int j = 0; j < ROWS; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int i0 = (k + j) & 1, qa = 4 * j + i0, qb = qa + 2, pi = 2 * j + k;
                wl[pi] = x2_pack(fw[0][qa], fw[0][qb]);
                wr[pi] = x2_pack(fw[1][qa], fw[1][qb]);
                wu[pi] = x2_pack(fw[2][qa], fw[2][qb]);
                wd[pi] = x2_pack(fw[3][qa], fw[3][qb]);
                inv[pi] = x2_pack(finv[qa], finv[qb]);
                rc[pi] = 0;
                dv[pi] = 0;
            }
    }
    // every word of the correction image starts at 0 (rows' padding included)
    for (int i = threadIdx.x; i < 2 * EY * WP; i += NT) (&T.d[0][0][0])[i] = 0.0f;
    __syncthreads();
    const double cdiv = P.cdiv, factor = P.factor;
    const f32x2 wgt2 = x2_pack(wgt, wgt), omw2 = x2_pack(omw1, omw1), one2 = x2_pack(P.one, P.one);
    // Shared-memory words of the neighbours in other blocks, clamped inside the image for the outermost blocks.
    // The one-word neighbours left and right of the block come from 8-byte loads of the aligned word pair that
    // holds them (the left one is the pair's high word, the right one its low word): a warp's side loads are
    // then consecutive 8-byte words, free of bank conflicts like the pair loads.
    const int cl = max(2 * bx - 2, 0), cr = min(2 * bx + 2, W2 - 2);
    const int ru = max(y0 - 1, 0), rd = min(y0 + ROWS, EY - 1);
    // most central ring among the block's cells
    const int bmax = min(min(x0 + 3, EX - 1 - x0), min(y0 + ROWS - 1, EY - 1 - y0));
    // Half-sweep of colour K01: the pairs 2 j + K01 of every row j, neighbours of the other colour: above and
    // below from the pairs of the rows beside it (shared memory past the block's edge rows), left and right
    // from the other pair of the same row and one word of shared memory past the block's edge columns.
    auto sweep = [&](auto kc) {
        constexpr int K01 = decltype(kc)::value;
        float(*Do)[WP] = T.d[1 - K01];
        const f32x2 upw = *reinterpret_cast<const f32x2*>(&Do[ru][2 * bx]);
        const f32x2 dnw = *reinterpret_cast<const f32x2*>(&Do[rd][2 * bx]);
        float side[ROWS];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const f32x2 w2 = *reinterpret_cast<const f32x2*>(&Do[y0 + j][((K01 + j) & 1) ? cr : cl]);
            side[j] = x2_lane(w2, ((K01 + j) & 1) ? 0 : 1);
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int pi = 2 * j + K01, po = 2 * j + (1 - K01);
            const f32x2 U = j > 0 ? dv[2 * (j - 1) + (1 - K01)] : upw;
            const f32x2 D = j < ROWS - 1 ? dv[2 * (j + 1) + (1 - K01)] : dnw;
            f32x2 Lf, Rt;
            if ((K01 + j) & 1) {  // cells 1 and 3: left (0, 2) in registers, right (2, 4)
                Lf = dv[po];
                Rt = x2_pack(x2_lane(dv[po], 1), side[j]);
            } else {  // cells 0 and 2: left (-1, 1), right (1, 3) in registers
                Lf = x2_pack(side[j], x2_lane(dv[po], 0));
                Rt = dv[po];
            }
            dv[pi] = oct_update(rc[pi], wl[pi], wr[pi], wu[pi], wd[pi], inv[pi], omw2, dv[pi], Lf, Rt, U, D, wgt2,
                                one2);
        }
        if (active) {
#pragma unroll
            for (int j = 0; j < ROWS; ++j) *reinterpret_cast<f32x2*>(&T.d[K01][y0 + j][2 * bx]) = dv[2 * j + K01];
        }
    };
    // FP64 residual of the live counted cells, rc = f32(cdiv r) on update cells, d = 0, and the CTA's norms over
    // its owned counted cells (fixed order; returned by thread 0).
    auto check = [&]() -> double2 {
        double ar = 0.0, ab = 0.0;
        float frc[NC];
        // A row's cells of p once for its four cells, under the row's branch (all rows at once, they spill).  Cells of
        // the outermost ring, whose neighbours lie outside the image, are not counted.
        const int left = x0 > 0 ? -1 : 0, right = x0 + 4 < EX ? 4 : 3;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
#pragma unroll
            for (int i = 0; i < 4; ++i) frc[4 * j + i] = 0.0f;
            if (!((fl >> (32 + 4 * j)) & 15ull)) continue;
            const int above = y0 + j > 0 ? j - 1 : j, below = y0 + j + 1 < EY ? j + 1 : j;
            double row[6];
            row[0] = T.p[pix(left, j)];
#pragma unroll
            for (int i = 0; i < 4; ++i) row[1 + i] = T.p[pix(i, j)];
            row[5] = T.p[pix(right, j)];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = 4 * j + i, pi = oct_pair(q), ln = oct_lane(q);
                double sum = (double)x2_lane(wl[pi], ln) * row[i];
                sum = sum + (double)x2_lane(wr[pi], ln) * row[i + 2];
                sum = sum + (double)x2_lane(wu[pi], ln) * T.p[pix(i, above)];
                sum = sum + (double)x2_lane(wd[pi], ln) * T.p[pix(i, below)];
                const double bb = T.b[pix(i, j)];
                const double r = bb - factor * (T.den[pix(i, j)] * row[i + 1] - sum);
                const bool counted = (fl >> (32 + q)) & 1ull;
                if (counted && ((fl >> q) & 1ull)) frc[q] = (float)(cdiv * r);
                if (counted && ((fl >> (48 + q)) & 1ull)) {
                    ar += r * r;
                    ab += bb * bb;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int qa = 4 * j + ((k + j) & 1);
                rc[2 * j + k] = x2_pack(frc[qa], frc[qa + 2]);
                dv[2 * j + k] = 0;
            }
        if (active) {
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                *reinterpret_cast<f32x2*>(&T.d[0][y0 + j][2 * bx]) = 0;
                *reinterpret_cast<f32x2*>(&T.d[1][y0 + j][2 * bx]) = 0;
            }
        }
        ar = warp_sum(ar);
        ab = warp_sum(ab);
        __shared__ double red_r[NT / 32], red_b[NT / 32];
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        if (lane == 0) {
            red_r[wid] = ar;
            red_b[wid] = ab;
        }
        __syncthreads();
        double2 out = make_double2(0.0, 0.0);
        if (threadIdx.x == 0) {
            for (int k = 0; k < NT / 32; ++k) {
                out.x += red_r[k];
                out.y += red_b[k];
            }
        }
        __syncthreads();
        return out;
    };
    const std::integral_constant<int, 0> c0{};
    const std::integral_constant<int, 1> c1{};

    __shared__ double2 s_sums[OCT_MAX_CTAS];
    unsigned iters = 0, seq = 0, checks = 0;  // exchanges and checks so far: their tags
    double2 part = check();
    if (threadIdx.x == 0) P.partials[rank] = part;
    bool ok = grid_barrier(P.barrier, nblocks, P.spin_limit);
    double r = ok ? ps_total_relative(P.partials, nblocks) : 0.0;
    const double r0v = r;
    bool pending = false;  // a check's sums, read with the next exchange
    unsigned checked = 0;  // iterations at the last check
    auto fetch = [&]() {
        return oct_fetch_sums<NT>(P.xch, checks, (int)nblocks, P.barrier, P.spin_limit, s_sums);
    };
    while (ok && (pending || (!(r <= P.tol) && iters < P.max_iters))) {
        unsigned todo = min(P.check_interval, P.max_iters - iters);
        iters += todo;
        bool converged = false;
        while (todo > 0) {
            const unsigned kk = min((unsigned)KMAX, todo);
            for (unsigned it = 0; it < kk; ++it) {
                if (bmax >= 1 + 2 * (int)it) {  // a cell of the block lies in the region still needed
                    if (base) sweep(c0);  // red ((x + y) odd) first
                    else sweep(c1);
                }
                __syncthreads();
                if (bmax >= 2 + 2 * (int)it) {
                    if (base) sweep(c1);
                    else sweep(c0);
                }
                __syncthreads();
            }
            todo -= kk;
            // Exchange the correction's halo.
            ++seq;
            ulonglong2* const at = part_of + (seq & 1) * XP;
            bool got = true;
            if (owned) {
#pragma unroll
                for (int i = 0; i < NPAIR; ++i)
                    xch_store(at + i * NBLK, __float_as_uint(x2_lane(dv[i], 0)), __float_as_uint(x2_lane(dv[i], 1)), seq);
            }
            if (pending) got = fetch();
            if (active && !owned) {
                ulonglong2 w[NPAIR];
                const bool from = part_of != nullptr;
                if (from) got = xch_poll(at, NBLK, seq, w, P.barrier, P.spin_limit) && got;
#pragma unroll
                for (int j = 0; j < ROWS; ++j)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        // an update cell's correction; every other cell's is 0 (its tile may not take part)
                        const int pi = 2 * j + k, qa = 4 * j + ((k + j) & 1);
                        const float a = from && ((upd_halo >> qa) & 1u) ? __uint_as_float((uint32_t)w[pi].x) : 0.0f;
                        const float b = from && ((upd_halo >> (qa + 2)) & 1u) ? __uint_as_float((uint32_t)w[pi].y) : 0.0f;
                        dv[pi] = x2_pack(a, b);
                        *reinterpret_cast<f32x2*>(&T.d[k][y0 + j][2 * bx]) = dv[pi];
                    }
            }
            ok = __syncthreads_and(got);
            if (!ok) break;
            if (pending) {
                pending = false;
                r = oct_total_relative(s_sums, (int)nblocks);
                if (r <= P.tol) {
                    converged = true;
                    iters = checked;
                    break;
                }
            }
        }
        if (!ok || converged) break;
        // p += d on every cell of the image (0 where the reference zeroes p): the halo's corrections are its owners'.
        if (active) {
#pragma unroll
            for (int q = 0; q < NC; ++q)
                T.p[pix(q & 3, q >> 2)] =
                    (upd_halo >> q) & 1u ? T.p[pix(q & 3, q >> 2)] + (double)x2_lane(dv[oct_pair(q)], oct_lane(q)) : 0.0;
        }
        __syncthreads();
        part = check();
        ++checks;
        checked = iters;
        if (threadIdx.x == 0) {
            ulonglong2* const sum = P.xch + ((checks & 1) * OCT_MAX_TILES + rank) * 2;
            xch_store(sum, part.x, checks);
            xch_store(sum + 1, part.y, checks);
            beat(rank);
        }
        if (iters < P.max_iters) {
            pending = true;
        } else {
            ok = __syncthreads_and(fetch());
            if (!ok) break;
            r = oct_total_relative(s_sums, (int)nblocks);
        }
    }
    if (ok && iters > 0 && owned)
#pragma unroll
        for (int q = 0; q < NC; ++q)
            if ((fl >> (48 + q)) & 1ull)
                L.x.at(gx0 + x0 + (q & 3), gy0 + y0 + (q >> 2)) = T.p[pix(q & 3, q >> 2)];
    if (ok && iters > 0)  // the tiles that took no part: p = 0, as on every cell that is not updated
        for (int q = (int)(nblocks + rank); q < P.ntiles; q += (int)nblocks) {
            const int ox = (list[q] % P.tiles_x) * TXo, oy = (list[q] / P.tiles_x) * TYo;
            for (int i = threadIdx.x; i < TXo * TYo; i += NT) {
                const int gx = ox + i % TXo, gy = oy + i / TXo;
                if (gx < L.nx && gy < L.ny) L.x.p[(size_t)gy * L.x.P + gx] = 0.0;
            }
        }
    if (rank == 0 && threadIdx.x == 0) {
        P.result->iterations = iters;
        P.result->converged = (ok && r <= P.tol) ? 1 : 0;
        P.result->error = ok ? 0 : 1;
        P.result->r0 = r0v;
        P.result->r1 = r;
    }
    return ok;
}

template <int EX, int EY, int KMAX, int NT, int ROWS>
__global__ void __launch_bounds__(NT, 1) k_gsmix_oct(PersistentParams P) {
    __shared__ unsigned short list[OCT_MAX_TILES];
    __shared__ int n;
    if (P.retry && P.result->error != 2) return;  // the launch before this one solved it
    oct_tiles<EX - 4 * KMAX, EY - 4 * KMAX, NT>(P, list, &n);
    if (n == 0 || n > (int)gridDim.x) {  // no water (b = 0: converged at once), or more tiles than CTAs
        if (blockIdx.x == 0 && threadIdx.x == 0) *P.result = SolveResult{0, n == 0 ? 1 : 0, n ? 2 : 0, 0, 0.0, 0.0};
        return;
    }
    if ((int)blockIdx.x < n) oct_solve<EX, EY, KMAX, NT, ROWS>(P, list, blockIdx.x, (unsigned)n);
}

// The reference's fixed-count f32 sweeps (gauss_seidel.wgsl:12-88, `iters`
// red-black iterations, red first) as ONE cooperative launch for grids of at
// most one tile per SM: a thread holds a 2 x 2 block of the tile and its halo.
// Per cell, with the reference's f32
// coefficients: update cells p = w (nume / den) + (1 - w) p, zero cells
// (air, fully solid, |den| < 1e-6) p = 0, the outermost ring untouched.  The
// owned cells are exchanged through L2 every KMAX iterations (alternating
// planes) and stored to `out` once no CTA may still be loading its first
// image from `out`: after an exchange, or a grid barrier of its own.
//
// Bound by the latency of the slowest warp between two block barriers, and by
// the exchanges (2.4 us each).  So: both cells of a colour side by side, no
// weights and no division in warps of standard cells, and no lane that divides
// by zero or divides a zero (the division's slow path: a warp with such a lane
// took 1000 cycles for a half-sweep, the others 200), and every load of the
// first image in flight at once.  20 iterations: 41.3 -> 30.4 us at 64 x 64,
// 44.0 -> 32.7 us at 256 x 256, 41.6 -> 33.0 us at 512 x 512 on tiles of
// 64 x 32 cells, and 20.0 and 21.5 us (64 x 64, 256 x 256) on the small tiles.
template <int EX, int EY>
struct Quad32Tile {
    static constexpr int W2 = EX / 2, NB = (EX / 2) * (EY / 2);
    static constexpr int WP = W2 % 16 == 4 ? W2 : W2 + ((4 - W2 % 16) + 16) % 16;
    float4 w[4][NB];
    float p[2][EY][WP];  // [k][y][x / 2], k = (x + y) & 1 in the image (k = 0: the tile's base colour)
};
struct Gs32Params {
    Level L;  // x = the pressure (read at the start, written at the end), b, ls, fu, fv
    PF xb[2];  // exchange planes
    int tiles_x, iters;
    float cdiv, weight;
    GridBarrier* barrier;
    long long spin_limit;
    int* err;  // set to 2 if a grid barrier timed out (reported with the TMA sweep's flag)
};
// Two cells of one colour.  general: some update cell of the warp is not standard (w = 1, den = 4: nume / 4 is
// nume * 0.25 exactly, without the weights and the division).
EFL_DEV void gs32_update2(bool general, float cb0, const float4* w0, float den0, float& p0, float l0, float r0, float u0,
                          float d0, unsigned upd0, unsigned zero0, float cb1, const float4* w1, float den1, float& p1,
                          float l1, float r1, float u1, float d1, unsigned upd1, unsigned zero1, float wgt, float omw) {
    float n0 = cb0, n1 = cb1;
    if (general) {
        const float4 a = *w0, b = *w1;
        n0 = n0 + a.x * l0;
        n1 = n1 + b.x * l1;
        n0 = n0 + a.y * r0;
        n1 = n1 + b.y * r1;
        n0 = n0 + a.z * u0;
        n1 = n1 + b.z * u1;
        n0 = n0 + a.w * d0;
        n1 = n1 + b.w * d1;
        n0 = div_zero(upd0 ? n0 : 1.0f, den0);
        n1 = div_zero(upd1 ? n1 : 1.0f, den1);
    } else {
        n0 = (((n0 + l0) + r0) + u0) + d0;
        n1 = (((n1 + l1) + r1) + u1) + d1;
        n0 = n0 * 0.25f;
        n1 = n1 * 0.25f;
    }
    const float v0 = wgt * n0 + omw * p0, v1 = wgt * n1 + omw * p1;
    p0 = upd0 ? v0 : (zero0 ? 0.0f : p0);
    p1 = upd1 ? v1 : (zero1 ? 0.0f : p1);
}
template <int EX, int EY, int KMAX, int NT>
__global__ void __launch_bounds__(NT, NT < 512 ? 2 : 1) k_gs32_quad(Gs32Params P) {
    static_assert((EX / 2) * (EY / 2) <= NT && NT % 32 == 0 && EX % 2 == 0 && EY % 2 == 0, "2 x 2 blocks");
    extern __shared__ __align__(16) unsigned char q32_raw[];
    Quad32Tile<EX, EY>& T = *reinterpret_cast<Quad32Tile<EX, EY>*>(q32_raw);
    constexpr int H = 2 * KMAX, W2 = EX / 2, NB = Quad32Tile<EX, EY>::NB, WP = Quad32Tile<EX, EY>::WP;
    constexpr int TXo = EX - 2 * H, TYo = EY - 2 * H;
    const Level& L = P.L;
    const int gx0 = (blockIdx.x % P.tiles_x) * TXo - H, gy0 = (blockIdx.x / P.tiles_x) * TYo - H;
    const unsigned nblocks = gridDim.x;
    const bool active = threadIdx.x < NB;
    const int bx = active ? (int)threadIdx.x % W2 : 0, by = active ? (int)threadIdx.x / W2 : 0;
    const int base = (gx0 + gy0) & 1;
    const bool owned = bx >= H / 2 && bx < (H + TXo) / 2 && by >= H / 2 && by < (H + TYo) / 2;
    const bool ring0x = bx == 0 || bx == W2 - 1, ring0y = by == 0 || by == EY / 2 - 1;
    float pv[4], cb[4], den[4];
    unsigned fl = 0;  // bit q: update; bit 4 + q: zero; bit 8 + q: live (in the domain, not the outer ring);
                      // bit 16 + q: owned and in the domain
    unsigned gen = 0;  // a live update cell that is not standard; then: one in the warp
    // Every load of the block first, at clamped places (three dependent rounds per cell otherwise).
    const int bgx = gx0 + 2 * bx, bgy = gy0 + 2 * by;
    float lv[4][4], fu[2][3], fv[3][2], xb0[4], bb[4];
    {
        const int xs[4] = {min(max(bgx - 1, 0), L.nx - 1), min(max(bgx, 0), L.nx - 1), min(max(bgx + 1, 0), L.nx - 1),
                           min(max(bgx + 2, 0), L.nx - 1)};
        const int ys[4] = {min(max(bgy - 1, 0), L.ny - 1), min(max(bgy, 0), L.ny - 1), min(max(bgy + 1, 0), L.ny - 1),
                           min(max(bgy + 2, 0), L.ny - 1)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if ((i == 1 || i == 2) || (j == 1 || j == 2)) lv[j][i] = L.ls.at(xs[i], ys[j]);
        const int fx[3] = {xs[1], min(max(bgx + 1, 0), L.nx), min(max(bgx + 2, 0), L.nx)};
        const int fy[3] = {ys[1], min(max(bgy + 1, 0), L.ny), min(max(bgy + 2, 0), L.ny)};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                xb0[2 * j + i] = L.x.at(xs[1 + i], ys[1 + j]);
                bb[2 * j + i] = L.b.at(xs[1 + i], ys[1 + j]);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                fu[j][i] = L.fu.at(fx[i], ys[1 + j]);
                fv[i][j] = L.fv.at(xs[1 + j], fy[i]);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int qx = q & 1, qy = q >> 1;
        const int gx = bgx + qx, gy = bgy + qy;
        const bool edge = (ring0x && (qx == (bx == 0 ? 0 : 1))) || (ring0y && (qy == (by == 0 ? 0 : 1)));
        float4 wk = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        pv[q] = 0.0f;
        cb[q] = 0.0f;
        den[q] = 1.0f;  // of every lane that divides: a zero would take the slow path
        if (active && (unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny) {
            pv[q] = xb0[q];
            if (owned) fl |= 1u << (16 + q);
            const float lij = lv[1 + qy][1 + qx];
            bool update = false;
            float dn = 0.0f;
            const float f[4] = {fu[qy][qx], fu[qy][qx + 1], fv[qy][qx], fv[qy + 1][qx]};
            if (lij < 0.0f && !(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
                cb[q] = P.cdiv * bb[q];
                const float ln[4] = {lv[1 + qy][qx], lv[1 + qy][qx + 2], lv[qy][1 + qx], lv[qy + 2][1 + qx]};
                const bool in[4] = {gx > 0, gx + 1 < L.nx, gy > 0, gy + 1 < L.ny};
                float wv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (!in[k]) continue;
                    if (ln[k] < 0.0f) {
                        dn += f[k];
                        wv[k] = f[k];
                    } else {
                        dn += f[k] * (1.0f - ln[k] / lij);
                    }
                }
                wk = make_float4(wv[0], wv[1], wv[2], wv[3]);
                update = !(fabsf(dn) < 1.0e-6f);
            }
            den[q] = update ? dn : 1.0f;
            if (!edge) fl |= (update ? 1u << q : 1u << (4 + q)) | (1u << (8 + q));
            if (!edge && update && !(wk.x == 1.0f && wk.y == 1.0f && wk.z == 1.0f && wk.w == 1.0f)) gen = 1u;
        }
        if (active) {
            T.w[q][threadIdx.x] = wk;
            T.p[(q == 0 || q == 3) ? 0 : 1][2 * by + qy][bx] = pv[q];
        }
    }
    __syncthreads();
    gen = __reduce_or_sync(0xffffffffu, gen);
    const float wgt = P.weight, omw = 1.0f - P.weight;
    const int t = active ? (int)threadIdx.x : 0;
    const int r0 = 2 * by, r1 = 2 * by + 1;
    const int bxl = bx > 0 ? bx - 1 : 0, bxr = bx < W2 - 1 ? bx + 1 : bx;
    const int rup = r0 > 0 ? r0 - 1 : 0, rdn = r1 < EY - 1 ? r1 + 1 : r1;
    const int bring = min(min(2 * bx + 1, EX - 2 * bx), min(2 * by + 1, EY - 2 * by)) - 1;
    // both cells of a colour side by side, stored under a predicate
    auto sweep_base = [&]() {  // cells 0 and 3; neighbours of the other colour
        float(*Po)[WP] = T.p[1];
        const float pl0 = Po[r0][bxl], pu0 = Po[rup][bx], pr3 = Po[r1][bxr], pd3 = Po[rdn][bx];
        gs32_update2(gen, cb[0], &T.w[0][t], den[0], pv[0], pl0, pv[1], pu0, pv[2], fl & 1u, fl & 0x10u, cb[3],
                     &T.w[3][t], den[3], pv[3], pv[2], pr3, pv[1], pd3, fl & 8u, fl & 0x80u, wgt, omw);
        if (fl & 0x100u) T.p[0][r0][bx] = pv[0];
        if (fl & 0x800u) T.p[0][r1][bx] = pv[3];
    };
    auto sweep_other = [&]() {  // cells 1 and 2; neighbours of the base colour
        float(*Po)[WP] = T.p[0];
        const float pr1 = Po[r0][bxr], pu1 = Po[rup][bx], pl2 = Po[r1][bxl], pd2 = Po[rdn][bx];
        gs32_update2(gen, cb[1], &T.w[1][t], den[1], pv[1], pv[0], pr1, pu1, pv[3], fl & 2u, fl & 0x20u, cb[2],
                     &T.w[2][t], den[2], pv[2], pl2, pv[3], pv[0], pd2, fl & 4u, fl & 0x40u, wgt, omw);
        if (fl & 0x200u) T.p[1][r0][bx] = pv[1];
        if (fl & 0x400u) T.p[1][r1][bx] = pv[2];
    };
    bool ok = true;
    int xch = 0;
    for (int done = 0; done < P.iters && ok;) {
        const int kk = min(KMAX, P.iters - done);
        for (int it = 0; it < kk; ++it) {
            if (bring + 1 >= 1 + 2 * it) {  // a cell of the block lies in the region still needed
                if (base) sweep_base();       // red ((x + y) odd) first
                else sweep_other();
            }
            __syncthreads();
            if (bring + 1 >= 2 + 2 * it) {
                if (base) sweep_other();
                else sweep_base();
            }
            __syncthreads();
        }
        done += kk;
        if (done < P.iters) {  // exchange the halo through L2 (alternating planes)
            const PF& xb = P.xb[xch++ & 1];
            if (owned) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if ((fl >> (16 + q)) & 1u)
                        __stcg(&xb.p[(size_t)(gy0 + 2 * by + (q >> 1)) * xb.P + gx0 + 2 * bx + (q & 1)], pv[q]);
            }
            ok = grid_barrier(P.barrier, nblocks, P.spin_limit);
            if (!ok) break;
            if (active && !owned) {
                float hv[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int gx = gx0 + 2 * bx + (q & 1), gy = gy0 + 2 * by + (q >> 1);
                    hv[q] = ((unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny)
                                ? __ldcg(&xb.p[(size_t)gy * xb.P + gx])
                                : 0.0f;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) pv[q] = hv[q];
                T.p[0][r0][bx] = pv[0];
                T.p[1][r0][bx] = pv[1];
                T.p[1][r1][bx] = pv[2];
                T.p[0][r1][bx] = pv[3];
            }
            __syncthreads();
        }
    }
    // every CTA has read its first image of x: an exchange said so already
    if (ok && xch == 0) ok = grid_barrier(P.barrier, nblocks, P.spin_limit);
    if (!ok && threadIdx.x == 0) atomicExch(P.err, 2);
    if (ok && owned) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if ((fl >> (16 + q)) & 1u) L.x.at(gx0 + 2 * bx + (q & 1), gy0 + 2 * by + (q >> 1)) = pv[q];
    }
}

template <int EX, int EY, int KMAX, int NT>
inline efl_status launch_gs32_quad(SolverWorkspace& ws, Gs32Params P, cudaStream_t stream, std::string* err) {
    constexpr int TXo = EX - 4 * KMAX, TYo = EY - 4 * KMAX;
    const int tiles_x = (P.L.nx + TXo - 1) / TXo, tiles_y = (P.L.ny + TYo - 1) / TYo;
    if (tiles_x * tiles_y > ws.num_sms) return EFL_ERR_STATE;
    P.tiles_x = tiles_x;
    const void* kern = (const void*)k_gs32_quad<EX, EY, KMAX, NT>;
    const size_t smem = sizeof(Quad32Tile<EX, EY>);
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return EFL_ERR_STATE;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return EFL_ERR_STATE;
        }
        attr_done[dev] = true;
    }
    if (cudaMemsetAsync(ws.barrier, 0, sizeof(GridBarrier), stream) != cudaSuccess) {
        *err = "barrier reset failed";
        return EFL_ERR_CUDA;
    }
    void* args[] = {&P};
    count_launch();
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(tiles_x * tiles_y), dim3(NT), args, smem, stream);
    if (e != cudaSuccess) {
        *err = std::string("cooperative launch of the fixed-count sweep failed: ") + cudaGetErrorString(e);
        return EFL_ERR_CUDA;
    }
    return EFL_OK;
}

// n fixed f32 red-black iterations at level 0 as one cooperative launch, when
// the grid fits one tile per SM: tiles of 32 x 16 cells, exchanged every 5
// iterations, where they do (256 x 256, 20 iterations: 21.5 us, against 32.7 us
// on the larger ones), else 64 x 32, every 4 (512 x 512: 33 us).  32 x 16 cells
// every 4, 6 and 7 iterations took 22.3, 23.0 and 22.4 us at 256 x 256.
// Two blocks of the small kernel fit an SM, so that simulations in flight together run side by side (three of
// 256 x 256: 45 us a frame; 54 us with one block per SM, 45 us on the larger tiles, whose frame alone takes 9 us more).
// EFL_ERR_STATE: it fits neither (use the TMA-streamed sweeps).
inline efl_status solve_gs32_persistent(SolverWorkspace& ws, const Level& L, const PF& xa, const PF& xb,
                                        float dx_scaled, float rho, float dt, float weight, uint32_t n,
                                        int* dev_err, cudaStream_t stream, std::string* err) {
    if (n == 0) return EFL_OK;
    if (!dev_err) return EFL_ERR_STATE;
    Gs32Params P;
    P.L = L;
    P.xb[0] = xa;
    P.xb[1] = xb;
    P.tiles_x = 0;
    P.iters = (int)n;
    P.cdiv = dx_scaled * dx_scaled * rho / dt;  // gauss_seidel.wgsl:58
    P.weight = weight;
    P.barrier = ws.barrier;
    P.spin_limit = ws.spin_limit > 0 ? ws.spin_limit : kBarrierSpinLimit;
    P.err = dev_err;
    const efl_status st = launch_gs32_quad<52, 36, 5, 480>(ws, P, stream, err);
    return st == EFL_ERR_STATE ? launch_gs32_quad<80, 48, 4, 960>(ws, P, stream, err) : st;
}

// Global-memory form of the same solve for grids the persistent scheme
// cannot hold (one launch per step of the algorithm).
struct MixPlanes {
    Plane<float4> w;
    PF inv, rc, d;
    Plane<double> den;
    Plane<unsigned char> mode;
};
// CG: the conjugate gradients imply a standard cell's coefficients and use none of a cell that is not counted.
template <bool CG>
__global__ void k_mix_coefficients(Level64 L, MixPlanes M) {
    const int gx = blockIdx.x * blockDim.x + threadIdx.x, gy = blockIdx.y * blockDim.y + threadIdx.y;
    if (gx >= L.nx || gy >= L.ny) return;
    unsigned char m = MODE_ZERO;
    double den = 0.0;
    float inv = 0.0f;
    float4 wk = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float phi = L.ls.at(gx, gy);
    if (phi < 0.0f) {
        const float f[4] = {L.fu.at(gx, gy), L.fu.at(gx + 1, gy), L.fv.at(gx, gy), L.fv.at(gx, gy + 1)};
        if (!(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
            m |= MODE_COUNTED;
            const int ox[4] = {-1, 1, 0, 0}, oy[4] = {0, 0, -1, 1};
            float wv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int jx = gx + ox[q], jy = gy + oy[q];
                if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
                    const float level = L.ls.at(jx, jy);
                    if (level < 0.0f) {
                        den += (double)f[q];
                        wv[q] = f[q];
                    } else {
                        den += (double)f[q] * (1.0 - (double)level / (double)phi);
                    }
                }
            }
            wk = make_float4(wv[0], wv[1], wv[2], wv[3]);
            if (!(fabs(den) < (double)1.0e-6f)) {
                m = (unsigned char)((m & MODE_COUNTED) | MODE_UPDATE);
                inv = (float)(1.0 / den);
                if (wk.x == 1.0f && wk.y == 1.0f && wk.z == 1.0f && wk.w == 1.0f) m |= MODE_STD;
            }
        }
    }
    M.mode.at(gx, gy) = m;
    if (CG && ((m & MODE_STD) || !(m & MODE_COUNTED))) return;
    M.den.at(gx, gy) = den;
    M.w.at(gx, gy) = wk;
    if (!CG) M.inv.at(gx, gy) = inv;
}
__global__ void __launch_bounds__(NORM_THREADS) k_mix_residual(Level64 L, MixPlanes M, double cdiv, double factor,
                                                               double2* partials) {
    __shared__ double sr[NORM_THREADS / 32], sb[NORM_THREADS / 32];
    double ar = 0.0, ab = 0.0;
    const int n = L.nx * L.ny;
    for (int i = blockIdx.x * NORM_THREADS + threadIdx.x; i < n; i += gridDim.x * NORM_THREADS) {
        const int y = i / L.nx, x = i - y * L.nx;
        const unsigned char m = M.mode.at(x, y);
        float rcv = 0.0f;
        if (m & MODE_COUNTED) {
            const float4 wk = M.w.at(x, y);
            double sum = (double)wk.x * L.x.ld(x - 1, y);
            sum = sum + (double)wk.y * L.x.ld(x + 1, y);
            sum = sum + (double)wk.z * L.x.ld(x, y - 1);
            sum = sum + (double)wk.w * L.x.ld(x, y + 1);
            const double bb = L.b.at(x, y);
            const double r = bb - factor * (M.den.at(x, y) * L.x.at(x, y) - sum);
            if (m & MODE_UPDATE) rcv = (float)(cdiv * r);
            ar += r * r;
            ab += bb * bb;
        }
        M.rc.at(x, y) = rcv;
        M.d.at(x, y) = 0.0f;
    }
    ar = warp_sum(ar);
    ab = warp_sum(ab);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        sr[wid] = ar;
        sb[wid] = ab;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double tr = 0.0, tb = 0.0;
        for (int k = 0; k < NORM_THREADS / 32; ++k) {
            tr += sr[k];
            tb += sb[k];
        }
        partials[blockIdx.x] = make_double2(tr, tb);
    }
}
__global__ void k_mix_sweep(MixPlanes M, int nx, int ny, float w, int color) {
    const int tx = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int x = 2 * tx + ((y + color) & 1);
    if (x >= nx || y >= ny) return;
    if (!(M.mode.at(x, y) & MODE_UPDATE)) return;
    const float4 wk = M.w.at(x, y);
    float nume = M.rc.at(x, y);
    nume = nume + wk.x * M.d.ld(x - 1, y);
    nume = nume + wk.y * M.d.ld(x + 1, y);
    nume = nume + wk.z * M.d.ld(x, y - 1);
    nume = nume + wk.w * M.d.ld(x, y + 1);
    M.d.at(x, y) = w * (nume * M.inv.at(x, y)) + (1.0f - w) * M.d.at(x, y);
}
__global__ void k_mix_apply(Level64 L, MixPlanes M) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= L.nx || y >= L.ny) return;
    double& pv = L.x.at(x, y);
    pv = (M.mode.at(x, y) & MODE_UPDATE) ? pv + (double)M.d.at(x, y) : 0.0;
}

// ---------------------------------------------------------------------------
// Fixed-count f32 sweeps (the reference's mode) as tiled, temporally blocked
// launches: each CTA loads its tile plus a halo of 2K cells, builds the
// per-cell coefficients of gauss_seidel.wgsl:44-80 in the reference's f32
// operation order (c*div, denom, neighbour weights), runs K red-black
// iterations from shared memory and writes its owned cells to the other
// buffer of a ping-pong pair.  Bit-identical to K global red/black sweeps.
template <int EX, int EY>
struct GsTile32 {
    static constexpr int W2 = EX / 2;
    static constexpr int N2 = W2 * EY;
    float p[2][N2];
    float cb[2][N2];
    float den[2][N2];
    float4 w[2][N2];
    unsigned char mode[2][N2];
};
constexpr int GT_THREADS = 256;

template <int EX, int EY, int K>
__global__ void __launch_bounds__(GT_THREADS) k_gs32_tile(Level L, PF out, float dx_scaled, float rho, float dt,
                                                          float weight, int tiles_x, int iters) {
    extern __shared__ __align__(16) unsigned char gt_raw[];
    GsTile32<EX, EY>& T = *reinterpret_cast<GsTile32<EX, EY>*>(gt_raw);
    constexpr int H = 2 * K, W2 = EX / 2, TX = EX - 2 * H, TY = EY - 2 * H;
    const int gx0 = (blockIdx.x % tiles_x) * TX - H, gy0 = (blockIdx.x / tiles_x) * TY - H;
    const int base = (gx0 + gy0) & 1;
    const float cdiv = dx_scaled * dx_scaled * rho / dt;  // gauss_seidel.wgsl:58
    for (int i = threadIdx.x; i < EX * EY; i += GT_THREADS) {
        const int ly = i / EX, lx = i - ly * EX;
        const int gx = gx0 + lx, gy = gy0 + ly;
        const int c = (base + lx + ly) & 1, k = ly * W2 + (lx >> 1);
        unsigned char m = MODE_SKIP;
        float den = 0.0f, cb = 0.0f, pv = 0.0f;
        float4 wk = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if ((unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny) {
            pv = L.x.at(gx, gy);
            const float lij = L.ls.at(gx, gy);
            bool update = false;
            if (lij < 0.0f) {
                const float f[4] = {L.fu.at(gx, gy), L.fu.at(gx + 1, gy), L.fv.at(gx, gy), L.fv.at(gx, gy + 1)};
                if (!(f[0] == 0.0f && f[1] == 0.0f && f[2] == 0.0f && f[3] == 0.0f)) {
                    cb = cdiv * L.b.at(gx, gy);
                    const int ox[4] = {-1, 1, 0, 0}, oy[4] = {0, 0, -1, 1};
                    float wv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int jx = gx + ox[q], jy = gy + oy[q];
                        if ((unsigned)jx < (unsigned)L.nx && (unsigned)jy < (unsigned)L.ny) {
                            const float level = L.ls.at(jx, jy);
                            if (level < 0.0f) {
                                den += f[q];
                                wv[q] = f[q];
                            } else {
                                den += f[q] * (1.0f - level / lij);
                            }
                        }
                    }
                    wk = make_float4(wv[0], wv[1], wv[2], wv[3]);
                    update = !(fabsf(den) < 1.0e-6f);
                }
            }
            const bool ring = lx == 0 || ly == 0 || lx == EX - 1 || ly == EY - 1;
            if (!ring) m = update ? MODE_UPDATE : MODE_ZERO;
        }
        T.p[c][k] = pv;
        T.cb[c][k] = cb;
        T.den[c][k] = den;
        T.w[c][k] = wk;
        T.mode[c][k] = m;
    }
    __syncthreads();
    const float omw = 1.0f - weight;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int c = half == 0 ? 1 : 0, o = 1 - c;  // red ((x+y) odd) first
            constexpr int TOTAL = (EY - 2) * W2;
            for (int i = threadIdx.x; i < TOTAL; i += GT_THREADS) {
                const int ly = 1 + i / W2;
                const int k = ly * W2 + (i - (ly - 1) * W2);
                const unsigned char m = T.mode[c][k];
                if (m & MODE_UPDATE) {
                    const int odd = (base + ly + c) & 1;
                    const float4 wk = T.w[c][k];
                    float nume = T.cb[c][k];
                    nume = nume + wk.x * T.p[o][k - 1 + odd];
                    nume = nume + wk.y * T.p[o][k + odd];
                    nume = nume + wk.z * T.p[o][k - W2];
                    nume = nume + wk.w * T.p[o][k + W2];
                    const float pn = nume / T.den[c][k];
                    T.p[c][k] = weight * pn + omw * T.p[c][k];
                } else if (m & MODE_ZERO) {
                    T.p[c][k] = 0.0f;
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < TX * TY; i += GT_THREADS) {
        const int ly = H + i / TX, lx = H + i % TX;
        const int gx = gx0 + lx, gy = gy0 + ly;
        if ((unsigned)gx < (unsigned)L.nx && (unsigned)gy < (unsigned)L.ny)
            out.at(gx, gy) = T.p[(base + lx + ly) & 1][ly * W2 + (lx >> 1)];
    }
}

// n fixed f32 red-black iterations on level L, ping-ponging between L.x and
// `alt` (same extent and pitch); the result ends in L.x.
inline efl_status solve_gs32_tiled(const Level& L, const PF& alt, float dx_scaled, float rho, float dt, float weight,
                                   uint32_t n, cudaStream_t stream) {
    constexpr int K = 2, EX = 64 + 4 * K, EY = 32 + 4 * K;  // 64 x 32 owned, two CTAs per SM
    constexpr int TX = EX - 4 * K, TY = EY - 4 * K;
    const size_t smem = sizeof(GsTile32<EX, EY>);
    int dev = 0;
    cudaGetDevice(&dev);
    static bool attr_done[64] = {};
    if (dev < 0 || dev >= 64) return EFL_ERR_CUDA;
    if (!attr_done[dev]) {
        if (cudaFuncSetAttribute(k_gs32_tile<EX, EY, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return EFL_ERR_CUDA;
        attr_done[dev] = true;
    }
    const int tiles_x = (L.nx + TX - 1) / TX, tiles_y = (L.ny + TY - 1) / TY;
    Level cur = L;
    PF dst = alt;
    uint32_t launches = 0;
    for (uint32_t done = 0; done < n;) {
        const int k = (int)std::min<uint32_t>(K, n - done);
        k_gs32_tile<EX, EY, K><<<tiles_x * tiles_y, GT_THREADS, smem + count_launch(), stream>>>(
            cur, dst, dx_scaled, rho, dt, weight, tiles_x, k);
        PF prev = cur.x;
        cur.x = dst;
        dst = prev;
        done += (uint32_t)k;
        ++launches;
    }
    if (launches & 1) {  // result is in alt: copy back
        if (cudaMemcpy2DAsync(L.x.p, (size_t)L.x.P * 4, alt.p, (size_t)alt.P * 4, (size_t)L.nx * 4, L.ny,
                              cudaMemcpyDeviceToDevice, stream) != cudaSuccess)
            return EFL_ERR_CUDA;
    }
    return EFL_OK;
}

struct PersistentPlan {
    int tx = 0, ty = 0, kmax = 0, tiles_x = 0, tiles_y = 0;
    int threads = 0;
    size_t smem = 0;
    const void* kernel = nullptr;
    bool ok = false;
};

// One CTA of `threads` threads with `smem` bytes of dynamic shared memory resident per SM (registers and shared
// memory both; sets the kernel's shared-memory limit), checked once per kernel and device.
template <const void* (*KernelOf)()>
inline bool plan_resident(int threads, size_t smem) {
    int dev = 0;
    cudaGetDevice(&dev);
    static signed char state[64] = {};  // 0 unknown, 1 resident, -1 not
    if (dev < 0 || dev >= 64) return false;
    if (!state[dev]) {
        const void* k = KernelOf();
        int per_sm = 0;
        const bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem) == cudaSuccess &&
                        per_sm >= 1;
        cudaGetLastError();
        state[dev] = ok ? 1 : -1;
    }
    return state[dev] == 1;
}
template <int EX, int EY, int KMAX, int NT, int ROWS>
inline const void* oct_kernel() { return (const void*)k_gsmix_oct<EX, EY, KMAX, NT, ROWS>; }
// Plans for the paired-lane form (OctTile: three doubles and a float per cell of the image, and padding).  The launch holds the tiles with
// water only, which are not known on the host: a plan whose tiles do not all fit the device at once is followed by
// the next one, which runs if it found too many.
template <int EX, int EY, int KMAX, int NT, int ROWS>
inline bool try_plan_oct(const SolverWorkspace& ws, int nx, int ny, PersistentPlan* p) {
    const int tx = EX - 4 * KMAX, ty = EY - 4 * KMAX;
    p->kmax = KMAX;
    p->tx = tx;
    p->ty = ty;
    p->tiles_x = (nx + tx - 1) / tx;
    p->tiles_y = (ny + ty - 1) / ty;
    p->smem = sizeof(OctTile<EX, EY, ROWS>);
    p->kernel = (const void*)k_gsmix_oct<EX, EY, KMAX, NT, ROWS>;
    p->threads = NT;
    if ((int64_t)p->tiles_x * p->tiles_y > OCT_MAX_TILES || ws.num_sms > OCT_MAX_CTAS) return false;
    return p->ok = plan_resident<oct_kernel<EX, EY, KMAX, NT, ROWS>>(NT, p->smem);
}
inline std::vector<PersistentPlan> plan_oct(const SolverWorkspace& ws, int nx, int ny) {
    std::vector<PersistentPlan> v;
    auto add = [&](auto try_plan) {  // true: every tile fits, no further plan is needed
        PersistentPlan p;
        if (!try_plan(ws, nx, ny, &p)) return false;
        v.push_back(p);
        return p.tiles_x * p.tiles_y <= ws.num_sms;
    };
    if (add(try_plan_oct<OCT_SMALL>) ||             // 32 x 32 owned, 8 iterations between exchanges
        add(try_plan_oct<OCT_MEDIUM>) ||            // 64 x 32, 4
        add(try_plan_oct<80, 72, 4, 384, 4>)) {}    // 64 x 56, 4 (1.63 us per iteration)
    return v;
}

// The exchanges' words for the largest of the plans (never inside a capture: the solve ends in a synchronisation).
inline bool oct_reserve(SolverWorkspace& ws, size_t bytes) {
    if (ws.xch_bytes >= bytes) return true;
    cudaFree(ws.xch);
    ws.xch = nullptr;
    ws.xch_bytes = 0;
    if (cudaMalloc(&ws.xch, bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    ws.xch_bytes = bytes;
    return true;
}

// Tolerance-driven solve, one cooperative launch.  EFL_ERR_STATE: the grid
// does not fit the persistent scheme.
inline efl_status solve_gsmix_persistent(SolverWorkspace& ws, const Level64& L, const Uniform& U,
                                         float weight, double tol, uint32_t max_iters, uint32_t check_interval,
                                         cudaStream_t stream, SolveResult* out, std::string* err) {
    const std::vector<PersistentPlan> plans = plan_oct(ws, L.nx, L.ny);
    if (plans.empty()) return EFL_ERR_STATE;
    PersistentParams P{};
    P.L = L;
    const double dx = (double)U.dx;
    P.cdiv = dx * dx * (double)U.rho / (double)U.dt;
    P.factor = (double)U.dt / (double)U.rho / dx / dx;
    P.weight = (double)weight;
    P.tol = tol;
    P.max_iters = max_iters;
    P.check_interval = std::max<uint32_t>(1, check_interval);
    P.partials = ws.partials;
    P.barrier = ws.barrier;
    P.result = ws.result;
    P.spin_limit = ws.spin_limit > 0 ? ws.spin_limit : kBarrierSpinLimit;
    size_t bytes = 0;
    for (const PersistentPlan& plan : plans)
        bytes = std::max(bytes, oct_xch_bytes(std::min(plan.tiles_x * plan.tiles_y, ws.num_sms), plan.tx * plan.ty));
    if (!oct_reserve(ws, bytes)) {
        *err = "out of device memory for the solve's exchanges";
        return EFL_ERR_OUT_OF_MEMORY;
    }
    P.xch = ws.xch;
    P.one = 1.0f;
    P.wet = ws.wet;
    P.wet_w = (L.nx + 31) / 32;
    k_wet_blocks<<<dim3(P.wet_w, (L.ny + 7) / 8), dim3(32, 8), count_launch(), stream>>>(L.ls, ws.wet);
    if (cudaMemsetAsync(ws.barrier, 0, sizeof(GridBarrier), stream) != cudaSuccess) {
        *err = "barrier reset failed";
        return EFL_ERR_CUDA;
    }
    for (const PersistentPlan& plan : plans) {
        P.tiles_x = plan.tiles_x;
        P.ntiles = plan.tiles_x * plan.tiles_y;
        P.retry = &plan != &plans[0];
        void* args[] = {&P};
        count_launch();
        const cudaError_t e = cudaLaunchCooperativeKernel(plan.kernel, dim3(std::min(P.ntiles, ws.num_sms)),
                                                          dim3(plan.threads), args, plan.smem, stream);
        if (e != cudaSuccess) {
            *err = std::string("cooperative launch of the mixed solver failed: ") + cudaGetErrorString(e);
            return EFL_ERR_CUDA;
        }
    }
    if (cudaMemcpyAsync(ws.h_state, ws.state, sizeof(SolveState), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess) {
        *err = std::string("mixed solver failed: ") + cudaGetErrorString(cudaGetLastError());
        return EFL_ERR_CUDA;
    }
    *out = ws.h_state->result;
    const int waits = ws.h_state->barrier.error;
    if (out->error == 2) return EFL_ERR_STATE;  // more tiles with water than the device holds
    if (out->error || waits) {
        *err = waits == 2 ? "mixed solver: a halo exchange timed out" : "mixed solver: a grid barrier timed out";
        return EFL_ERR_CUDA;
    }
    return EFL_OK;
}

// The same solve with global-memory kernels and a host loop (grids beyond the
// persistent scheme).  M must hold planes of the level's extent.
inline efl_status solve_gsmix_global(SolverWorkspace& ws, const Level64& L, const MixPlanes& M, const Uniform& U,
                                     float weight, double tol, uint32_t max_iters, uint32_t check_interval,
                                     cudaStream_t stream, SolveResult* out, std::string* err) {
    const dim3 b(32, 8);
    const dim3 g((L.nx + 31) / 32, (L.ny + 7) / 8);
    const dim3 gh(((L.nx + 1) / 2 + 31) / 32, (L.ny + 7) / 8);
    const double dx = (double)U.dx;
    const double cdiv = dx * dx * (double)U.rho / (double)U.dt;
    const double factor = (double)U.dt / (double)U.rho / dx / dx;
    const int nblocks = std::min(ws.max_blocks, std::max(1, (L.nx * L.ny + NORM_THREADS - 1) / NORM_THREADS));
    k_mix_coefficients<false><<<g, b, count_launch(), stream>>>(L, M);
    auto residual = [&](double* rel) -> efl_status {
        k_mix_residual<<<nblocks, NORM_THREADS, count_launch(), stream>>>(L, M, cdiv, factor, ws.partials);
        std::vector<double2> h(nblocks);
        if (cudaMemcpyAsync(h.data(), ws.partials, nblocks * sizeof(double2), cudaMemcpyDeviceToHost, stream) !=
                cudaSuccess ||
            cudaStreamSynchronize(stream) != cudaSuccess) {
            *err = std::string("mixed solver (global): ") + cudaGetErrorString(cudaGetLastError());
            return EFL_ERR_CUDA;
        }
        double r = 0.0, bb = 0.0;
        for (int i = 0; i < nblocks; ++i) {
            r += h[i].x;
            bb += h[i].y;
        }
        *rel = bb > 0.0 ? std::sqrt(r) / std::sqrt(bb) : (r > 0.0 ? INFINITY : 0.0);
        return EFL_OK;
    };
    double rel;
    efl_status st = residual(&rel);
    if (st != EFL_OK) return st;
    out->r0 = rel;
    uint32_t iters = 0;
    const uint32_t chk = std::max<uint32_t>(1, check_interval);
    while (!(rel <= tol) && iters < max_iters) {
        const uint32_t n = std::min(chk, max_iters - iters);
        for (uint32_t it = 0; it < n; ++it) {
            k_mix_sweep<<<gh, b, count_launch(), stream>>>(M, L.nx, L.ny, weight, 1);
            k_mix_sweep<<<gh, b, count_launch(), stream>>>(M, L.nx, L.ny, weight, 0);
        }
        k_mix_apply<<<g, b, count_launch(), stream>>>(L, M);
        iters += n;
        st = residual(&rel);
        if (st != EFL_OK) return st;
    }
    out->iterations = iters;
    out->r1 = rel;
    out->converged = rel <= tol ? 1 : 0;
    out->error = 0;
    return EFL_OK;
}

}  // namespace efl
