// efl_gang.cuh — the tolerance-driven pressure solves of many independent simulations in ONE cooperative launch of one
// CTA per SM, each simulation solved by a gang of CTAs.
//
// A gang is as many CTAs as the simulation has tiles with water (64 x 32 cells, oct_solve), so a simulation keeps its
// tiles in shared memory and registers for the whole solve, exchanges halos with its own CTAs only, and frees them
// when it has converged, while the other gangs go on at their own pace.  CTAs without a gang are idle; whenever one
// becomes idle, the largest simulation that fits the idle CTAs starts (a list in global memory behind a lock).  The
// streamed form (efl_batch.cuh) runs every simulation in lockstep, each round reading every active tile from L2 behind
// a barrier of the whole device: about 10 us per red-black iteration whatever the number of simulations left, against
// 0.9 us here.  64 x 32 tiles because of the throughput per SM, 2270 cells per us (32 x 32: 1480; 64 x 56: 2200, but
// 1.6 us per iteration and coarser tiles).  A step of 32 pools of 128^2 to 768^2: 78 ms (91 before the checks shared an
// exchange; then 134 with an exchange every 8 iterations instead of 4, by 4 x 4 blocks that spill).
//
// Each simulation's iterates and iteration count are those of its own solve.  Every wait is bounded: those of a gang
// by polls, an idle CTA's (for its next gang, which may take other simulations' whole solves, or for the lock) by polls
// in which no gang comes to its next residual check; gang_idle_limit gives a gang's own waits up to there time to run out
// first.  (A report per exchange instead cost 0.6 % of a step.)
#pragma once

#include "efl_solver.cuh"

namespace efl {

#define GANG_TILE OCT_MEDIUM
constexpr int GANG_THREADS = 480, GANG_TX = 64, GANG_TY = 32, GANG_K = 4;
constexpr int GANG_MAX_SIMS = 512, GANG_MAX_CTAS = 512;

struct GangSim {
    PersistentParams P;
};
struct GangState {  // zeroed before each launch
    unsigned lock;
    int arrived;    // CTAs that have been idle once
    int nidle;
    int started;    // simulations started or not schedulable
    int smallest;   // no simulation left has fewer tiles
    int error;      // a wait ran out
    unsigned beat;  // grows with all progress: CTAs that become idle, simulations started, residual checks
    unsigned taken[GANG_MAX_SIMS / 32];
    int idle[GANG_MAX_CTAS];
    int2 mail[GANG_MAX_CTAS];  // (simulation + 1, rank) for a CTA; x = 0: none yet, -1: leave
    int n[GANG_MAX_SIMS];      // tiles with water
};

EFL_DEV int gang_load(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Polls between two checks `interval` iterations apart: the exchanges' and a check's at most `limit` each.
inline long long gang_idle_limit(long long limit, unsigned interval) {
    const long long waits = (long long)interval / GANG_K + 3;
    return limit > (1ll << 62) / waits ? 1ll << 62 : limit * waits;
}
// A wait for other CTAs' progress: true while it may go on.
struct GangWait {
    volatile GangState* V;
    long long limit, spins = 0;
    unsigned seen;
    EFL_DEV GangWait(GangState* G, long long lim) : V(G), limit(lim), seen(V->beat) {}
    EFL_DEV bool poll() {
        if ((++spins & 1023) != 0 && spins < limit) return true;
        if (V->error) return false;
        const unsigned now = V->beat;
        if (now == seen) return spins < limit;
        seen = now;
        spins = 0;
        return true;
    }
};
// oct_solve's report of a residual check.
struct GangBeat {
    GangState* G;
    EFL_DEV void operator()(unsigned rank) const {
        if (rank == 0) atomicAdd(&G->beat, 1u);
    }
};

// Starts simulations while one fits the idle CTAs; lets the idle CTAs go when none is left.  Under the lock.
EFL_DEV void gang_schedule(GangState* G, int ns) {
    volatile GangState* V = G;
    int nidle = V->nidle, started = V->started, smallest = V->smallest;
    while (started < ns && nidle >= smallest) {
        int best = -1, bn = 0;
        smallest = 1 << 30;
#pragma unroll 8
        for (int i = 0; i < ns; ++i) {
            const int n = __ldcg(&G->n[i]);
            const bool left = !((__ldcg(&G->taken[i >> 5]) >> (i & 31)) & 1u);
            if (left && n < smallest) smallest = n;
            if (left && n <= nidle && n > bn) {
                bn = n;
                best = i;
            }
        }
        if (best < 0) break;
        V->taken[best >> 5] = V->taken[best >> 5] | (1u << (best & 31));
        __threadfence();
        ++started;
        atomicAdd(&G->beat, 1u);
        for (int r = 0; r < bn; ++r) {
            const int c = V->idle[--nidle];
            V->mail[c].y = r;
            __threadfence();
            V->mail[c].x = best + 1;
        }
    }
    if (started == ns)
        while (nidle > 0) V->mail[V->idle[--nidle]].x = -1;
    V->nidle = nidle;
    V->started = started;
    V->smallest = smallest;
}

// The calling CTA (its first thread) joins the idle ones and waits for its next gang: (simulation, rank), or x < 0.
EFL_DEV int2 gang_next(GangState* G, int ns, bool first, long long limit) {
    volatile GangState* V = G;
    for (GangWait w(G, limit); atomicCAS(&G->lock, 0u, 1u) != 0u;)
        if (!w.poll()) {
            atomicExch(&G->error, 1);
            return make_int2(-1, 0);
        }
    __threadfence();
    atomicAdd(&G->beat, 1u);
    V->idle[V->nidle] = (int)blockIdx.x;
    V->nidle = V->nidle + 1;
    if (first) V->arrived = V->arrived + 1;
    if (V->arrived == (int)gridDim.x) gang_schedule(G, ns);  // every simulation's tile count is known from here on
    __threadfence();
    atomicExch(&G->lock, 0u);
    int sim = 0;
    for (GangWait w(G, limit); (sim = gang_load(&G->mail[blockIdx.x].x)) == 0; __nanosleep(100))
        if (!w.poll()) {
            atomicExch(&G->error, 1);
            return make_int2(-1, 0);
        }
    const int rank = V->mail[blockIdx.x].y;
    V->mail[blockIdx.x].x = 0;
    return make_int2(sim > 0 ? sim - 1 : -1, rank);
}

__global__ void __launch_bounds__(GANG_THREADS, 1) k_batch_gang(const GangSim* sims, int ns, GangState* G,
                                                                long long limit) {
    __shared__ unsigned short list[OCT_MAX_TILES];
    __shared__ int n;
    __shared__ int2 job;
    __shared__ __align__(16) unsigned char raw[sizeof(GangSim)];
    const GangSim& S = *reinterpret_cast<const GangSim*>(raw);
    auto load = [&](int i) {
        static_assert(sizeof(GangSim) % 4 == 0, "copied by words");
        __syncthreads();
        for (int k = threadIdx.x; k < (int)sizeof(GangSim) / 4; k += GANG_THREADS)
            reinterpret_cast<unsigned*>(raw)[k] = reinterpret_cast<const unsigned*>(&sims[i])[k];
        __syncthreads();
        oct_tiles<GANG_TX, GANG_TY, GANG_THREADS>(S.P, list, &n);
    };
    for (int i = (int)blockIdx.x; i < ns; i += (int)gridDim.x) {
        load(i);
        if (threadIdx.x == 0) {
            // No water: converged at once.  More tiles than CTAs: left to the caller (error 2).
            const bool fits = n > 0 && n <= (int)gridDim.x;
            if (!fits) {
                *S.P.result = SolveResult{0, n == 0 ? 1 : 0, n ? 2 : 0, 0, 0.0, 0.0};
                atomicOr(&G->taken[i >> 5], 1u << (i & 31));
                atomicAdd(&G->started, 1);
            }
            __stcg(&G->n[i], n);
            __threadfence();
        }
    }
    bool first = true;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) job = gang_next(G, ns, first, limit);
        first = false;
        __syncthreads();
        const int2 j = job;
        if (j.x < 0) return;
        load(j.x);
        if (!oct_solve<GANG_TILE>(S.P, list, (unsigned)j.y, (unsigned)n, GangBeat{G})) {
            if (threadIdx.x == 0) atomicExch(&G->error, 1);
            return;
        }
    }
}

}  // namespace efl
