/*
 * work_share.cuh - how the persistent warps of the dynamic transport kernels
 * share the packets of a run: the packet queue and, once it is empty, the
 * packets still in flight.
 *
 * What bounds the end of a run is issue slots spent on nearly empty warps.
 * When the queue runs dry every warp holds up to 32 packets whose remaining
 * lives differ by two orders of magnitude; the few long ones are left one or
 * two to a warp, and all those warps compete for the SM's four schedulers
 * with 1 to 3 of 32 lanes active.  So the warps of a block merge their
 * packets as they thin out: a warp whose packets fit into the idle lanes of
 * the block's other warps leaves them in shared memory and ends.  Nothing
 * waits: the exchange is tried between steps and skipped when another warp
 * holds it.  A packet's state moves as a whole, so its path and the integer
 * tallies do not change.
 *
 * With the queue rule below: 1e4 packets of the slab (EXACT) 0.96 -> 0.65
 * ms, 1e6 (FAST) 1.70 -> 1.42 ms, 1e6 packets of the skin stack (FAST) 9.65
 * -> 7.5 ms, 1e7 49.2 -> 45.9 ms, 2e6 (EXACT) 31.1 -> 25.8 ms; 1e6 packets of
 * the skin and vessel voxels (FAST) 6.1 -> 5.8 ms.
 */
#pragma once
#include <cstdint>

#define WS_FULL 0xffffffffu

/* Copies a packet's state to or from one slot of the exchange, word by word. */
struct WsSave {
    uint32_t *at;
    __device__ __forceinline__ void word(uint32_t v) { *at = v; at += 32; }
    __device__ __forceinline__ void operator()(const float &v) { word(__float_as_uint(v)); }
    __device__ __forceinline__ void operator()(const int &v) { word((uint32_t)v); }
    __device__ __forceinline__ void operator()(const uint32_t &v) { word(v); }
    __device__ __forceinline__ void operator()(const uint64_t &v) { word((uint32_t)v); word((uint32_t)(v >> 32)); }
};
struct WsLoad {
    const uint32_t *at;
    __device__ __forceinline__ uint32_t word() { uint32_t v = *at; at += 32; return v; }
    __device__ __forceinline__ void operator()(float &v) { v = __uint_as_float(word()); }
    __device__ __forceinline__ void operator()(int &v) { v = (int)word(); }
    __device__ __forceinline__ void operator()(uint32_t &v) { v = word(); }
    __device__ __forceinline__ void operator()(uint64_t &v) {
        uint32_t lo = word();
        v = ((uint64_t)word() << 32) | lo;
    }
};

/* KEEP and SHARE by how much the kernel's steps diverge.  Layered: 1 and 8
   (four warps of an SM in the shortest runs); voxelized, where the lanes
   split between flights and walls: 2 and 2 (16 warps).  5e3 packets of the
   voxel grid with 1 and 1000 (all lanes of a warp) 2.1 ms, with 2 and 2 1.25
   ms (1.23 before warps merged); 3e3 of the slab with 1000 0.33, with 8 0.30
   ms (0.55 before). */
template <int WORDS, int WARPS, int KEEP, int SHARE>
struct WsExchange {
    uint32_t words[WORDS][32];
    int lock;          /* 1 while a warp uses the exchange; only ever tried */
    int count;         /* packets in it */
    int alive;         /* warps that have not left */
    int idle[WARPS];   /* idle lanes of the warps that have found the queue empty */
};

/* To be followed by a block barrier. */
template <int WORDS, int WARPS, int KEEP, int SHARE>
static __device__ __forceinline__ void ws_init(WsExchange<WORDS, WARPS, KEEP, SHARE> &e) {
    if (threadIdx.x < WARPS) e.idle[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        e.lock = 0;
        e.count = 0;
        e.alive = (int)(blockDim.x >> 5);
    }
}

/* A warp that leaves without its packets (deadline, abort). */
template <int WORDS, int WARPS, int KEEP, int SHARE>
static __device__ __forceinline__ void ws_leave(WsExchange<WORDS, WARPS, KEEP, SHARE> &e) {
    if ((threadIdx.x & 31u) == 0) *(volatile int *)&e.idle[threadIdx.x >> 5] = 0;
}

/* One try at the exchange by a warp (all lanes) that has found the queue
   empty.  Takes packets that another warp left into idle lanes; or, when
   there are none and the block's other warps have idle lanes for all of this
   warp's packets, leaves them there.  Idle lanes only grow by then, apart
   from what is taken here under the lock, so packets left are taken at the
   other warps' next try.  The last KEEP warps of a block keep what they
   have: a few warps on an SM do not yet slow one another, and fuller ones
   diverge more.  False: the warp has no packets and ends. */
template <int WORDS, int WARPS, int KEEP, int SHARE, class Visit>
static __device__ __forceinline__ bool ws_share(WsExchange<WORDS, WARPS, KEEP, SHARE> &e, bool &active, const Visit &visit) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t mask = __ballot_sync(WS_FULL, active);
    const int n = __popc(mask);
    if (n == 32) return true;
    int got = 0;
    if (lane == 0) {
        *(volatile int *)&e.idle[warp] = 32 - n;
        got = atomicCAS(&e.lock, 0, 1) == 0 ? 1 : 0;
    }
    got = __shfl_sync(WS_FULL, got, 0);
    if (!got) return true;
    __threadfence_block();
    bool stay = true;
    const int there = *(volatile int *)&e.count;
    if (there > 0) {
        const int take = min(there, 32 - n);
        const int rank = __popc(~mask & below);
        if (!active && rank < take) {
            WsLoad load{&e.words[0][there - 1 - rank]};
            visit(load);
            active = true;
        }
        __syncwarp();
        if (lane == 0) {
            *(volatile int *)&e.count = there - take;
            *(volatile int *)&e.idle[warp] = 32 - n - take;
        }
    } else {
        int room = (lane < WARPS && lane != warp) ? *(volatile int *)&e.idle[lane] : 0;
        room = __reduce_add_sync(WS_FULL, room);
        const int alive = *(volatile int *)&e.alive;
        if (n == 0 || (n <= room && alive > KEEP)) {
            if (active) {
                WsSave save{&e.words[0][__popc(mask & below)]};
                visit(save);
                active = false;
            }
            __syncwarp();
            if (lane == 0) {
                *(volatile int *)&e.count = n;
                *(volatile int *)&e.idle[warp] = 0;
                *(volatile int *)&e.alive = alive - 1;
            }
            stay = false;
        }
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) atomicExch(&e.lock, 0);
    return stay;
}

/* Whether this lane takes packets: in runs too short to fill one in SHARE
   warps of the grid, only an even share of a warp's lanes do. */
template <int WORDS, int WARPS, int KEEP, int SHARE>
static __device__ __forceinline__ bool ws_takes(const WsExchange<WORDS, WARPS, KEEP, SHARE> &, uint64_t N,
                                                uint32_t fixed, uint32_t warps) {
    return fixed != 0 || (threadIdx.x & 31u) <= N / (warps / (uint32_t)SHARE + 1u);
}

/* The next packets for a warp with `need` idle lanes: [first, end).  With a
   fixed item size, that many.  Else a quarter of an even share of the
   packets left at the warp's last visit, at most `most` (few visits in long
   runs) and at least the idle lanes: short runs fill warps instead of
   spreading single packets over all of them, and the last packets of a run
   go out one lane at a time. */
static __device__ __forceinline__ void ws_fetch(unsigned long long *queue, uint64_t N, uint32_t fixed,
                                                uint32_t most, uint32_t warps, int need, uint64_t &first,
                                                uint64_t &end) {
    const uint64_t left = first < N ? N - first : 0;
    uint64_t take = fixed;
    if (fixed == 0) {
        take = left / ((uint64_t)warps * 4u);
        take = take > most ? most : take;
        take = take < (uint64_t)need ? (uint64_t)need : take;
    }
    unsigned long long at = 0;
    if ((threadIdx.x & 31u) == 0) at = atomicAdd(queue, (unsigned long long)take);
    at = __shfl_sync(WS_FULL, at, 0);
    first = at;
    end = at + take < N ? at + take : N;
}
