/*
 * batched_kernel.cuh - thousands of independent single-layer simulations in
 * one persistent, work-stealing launch.
 *
 * The packets of all simulations are numbered consecutively (simulation s
 * owns [prefix[s], prefix[s+1])).  A work item is packets_per_item
 * consecutive packets; a warp takes items from a device-wide counter and
 * hands packets to its lanes one at a time: whenever lanes finish a packet,
 * a warp ballot gives them the next packets of the current item, taking a
 * new item when it runs out.  Lanes therefore stay busy until the last items
 * are gone, whatever the spread of packet lengths between simulations.
 *
 * Each packet owns the MWC stream derived from (seed, s, k) (batch_rng.h),
 * so the integer tallies are independent of the scheduling.  The physics of
 * a packet is the layered kernel's albedo-weight loop (mcml_boundary,
 * pf_sample, scatter_direction) on the simulation's three-layer table, with
 * a normally incident Line source and a radial reflectance tally at the top
 * surface; every simulation is statistically an mcml run of that shape.
 */
#pragma once
#include "mc_device.cuh"
#include "batch_rng.h"
#include "batch_launch.h"
#include "mcml_kernel.cuh"

namespace MCGB_NS {

/* Per-simulation table in the scratch buffer. */
struct __align__(16) BatchPrep {
    MlLayer L[3];
    float reflectance;      /* specular reflectance of the Line source */
    uint32_t sim;           /* the simulation: tables are in the order of batch_prep_kernel */
    float pad[2];
};
static_assert(sizeof(BatchPrep) <= MCGB_BATCH_PREP_BYTES,
              "a per-simulation table must fit the scratch record of batch_launch.h");

/* cos_critical / Fresnel at normal incidence in double precision, as the
   host-side packing of the layered simulator computes them
   (xopto/mcml/mclayer/layer.py:944-1007, mcutil/boundary.py:25-71). */
static __device__ __forceinline__ double cc_d(double n1, double n2) {
    return n1 > n2 ? sqrt(1.0 - (n2 / n1) * (n2 / n1)) : 0.0;
}

/* Bucket of a simulation by the most steps that its packets can live: a
   weight reaches the lottery after ln(1e4)/a steps of absorbed fraction a.
   Quarter octaves of 1/a, the longest first. */
constexpr int BATCH_BUCKETS = 128;
static __device__ __forceinline__ int batch_bucket(const McgbBatchSim &m) {
    float a = m.mua / (m.mua + m.mus);
    int life = cvt_int(fminf(-4.0f * __log2f(fmaxf(a, 1e-12f)), 126.0f));
    return BATCH_BUCKETS - 1 - clip_i(life, 0, BATCH_BUCKETS - 1);
}

/* One block: the simulations' order, packet prefix sums and the layer tables
   in that order.  The queue hands out the longest-lived packets first: taken
   in the caller's order, the last of them began when the rest was done, and
   the run waited for their 1e5 serial steps alone. */
__global__ void __launch_bounds__(1024)
batch_prep_kernel(const McgbBatchSim *sims, uint32_t S, uint64_t *prefix, BatchPrep *prep,
                  unsigned long long *queue) {
    __shared__ uint32_t start[BATCH_BUCKETS];
    __shared__ uint64_t part[32];
    const uint32_t tid = threadIdx.x, nt = blockDim.x, lane = tid & 31u;
    if (tid < BATCH_BUCKETS) start[tid] = 0;
    __syncthreads();
    for (uint32_t s = tid; s < S; s += nt) atomicAdd(&start[batch_bucket(sims[s])], 1u);
    __syncthreads();
    if (tid < 32) {
        uint32_t run = 0;
        for (int b = 0; b < BATCH_BUCKETS; b += 32) {
            uint32_t v = start[b + lane], sum = v;
            for (int d = 1; d < 32; d <<= 1) {
                uint32_t u = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += u;
            }
            start[b + lane] = run + sum - v;
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    __syncthreads();
    for (uint32_t s = tid; s < S; s += nt) {
        const McgbBatchSim m = sims[s];
        const uint32_t at = atomicAdd(&start[batch_bucket(m)], 1u);
        prefix[at] = m.num_packets;
        double mua = m.mua, mus = m.mus;
        double mut = mua + mus;
        float inv_mut = mut > 0.0 ? (float)(1.0 / mut) : __int_as_float(0x7f800000);
        float mua_inv_mut = mus == 0.0 ? 1.0f : (float)(mua * (mut > 0.0 ? 1.0 / mut : 0.0));
        float inf = __int_as_float(0x7f800000);
        BatchPrep p;
        McgbPf hg0 = {{0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, 0u, 0u, 0u};
        McgbPf hg1 = {{m.g, 0.0f, 0.0f, 0.0f, 0.0f}, 0u, 0u, 0u};
        p.L[0].g0 = make_float4(-inf, 0.0f, step_factor(inf), 1.0f);
        p.L[0].g1 = make_float4(m.n_above, 0.0f, 0.0f, 0.0f);
        p.L[0].g2 = make_float4((float)cc_d(m.n_above, m.n), 0.0f, 0.0f, 0.0f);
        pf_prepare(MCGB_PF_HG, hg0, p.L[0].pf0, p.L[0].pf1);
        p.L[1].g0 = make_float4(0.0f, m.thickness, step_factor(inv_mut), mua_inv_mut);
        p.L[1].g1 = make_float4(m.n, m.mua, m.mus, (float)cc_d(m.n, m.n_above));
        p.L[1].g2 = make_float4((float)cc_d(m.n, m.n_below), 0.0f, 0.0f, 0.0f);
        pf_prepare(MCGB_PF_HG, hg1, p.L[1].pf0, p.L[1].pf1);
#if MCGB_FAST_MATH
        /* the square inside the multiply-add, whatever the code around */
        p.L[1].pf0.y = __fmaf_rn(-m.g, m.g, 1.0f);
        p.L[1].pf0.z = __fmaf_rn(m.g, m.g, 1.0f);
#endif
        p.L[2].g0 = make_float4(m.thickness, inf, step_factor(inf), 1.0f);
        p.L[2].g1 = make_float4(m.n_below, 0.0f, 0.0f, (float)cc_d(m.n_below, m.n));
        p.L[2].g2 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        pf_prepare(MCGB_PF_HG, hg0, p.L[2].pf0, p.L[2].pf1);
        double r = ((double)m.n_above - m.n) / ((double)m.n_above + m.n);
        p.reflectance = (float)(r * r);
        p.sim = s;
        p.pad[0] = p.pad[1] = 0.0f;
        prep[at] = p;
    }
    __syncthreads();
    /* exclusive sums of the packet counts, one tile of the block at a time */
    uint64_t base = 0;
    for (uint32_t t = 0; t < S; t += nt) {
        const uint64_t v = t + tid < S ? prefix[t + tid] : 0ull;
        uint64_t sum = v;
        for (int d = 1; d < 32; d <<= 1) {
            uint64_t u = __shfl_up_sync(0xffffffffu, sum, d);
            if ((int)lane >= d) sum += u;
        }
        if (lane == 31) part[tid >> 5] = sum;
        __syncthreads();
        uint64_t before = 0, all = 0;
        for (uint32_t k = 0; k < nt / 32; ++k) {
            if (k < (tid >> 5)) before += part[k];
            all += part[k];
        }
        if (t + tid < S) prefix[t + tid] = base + before + sum - v;
        base += all;
        __syncthreads();
    }
    if (tid == 0) {
        prefix[S] = base;
        *queue = 0ull;
    }
}

/* A packet of the batch: always in the sample layer between steps. */
struct BatchPacket {
    f3 pos, dir;
    float w;
    uint32_t rec;   /* its simulation's table */
};

/* The sample layer's constants of a lane's simulation, kept in registers:
   one load per packet instead of three per step. */
struct BatchLayer {
    float factor, thickness, absorb;
    float4 pf0;
    float2 pf1;
    __device__ __forceinline__ void load(const BatchPrep &p) {
        const float4 g0 = p.L[1].g0, q = p.L[1].pf1;
        factor = g0.z;
        thickness = g0.y;
        absorb = g0.w;
        pf0 = p.L[1].pf0;
        pf1 = make_float2(q.x, q.y);
    }
};

typedef WsExchange<11, 8, 1, 8> BatchExchange;

template <class IO>
static __device__ __forceinline__ void batch_state(IO &io, BatchPacket &s, Rng &rng) {
    io(s.pos.x); io(s.pos.y); io(s.pos.z);
    io(s.dir.x); io(s.dir.y); io(s.dir.z);
    io(s.w); io(s.rec);
    io(rng.x); io(rng.a);
}

/* One step, as mcml_step_weight: the scattered direction is computed before
   it is known whether the path stays in the layer.  True when the packet
   ended.  What bounds a batch is issue, and for its longest packets (1e5
   steps) the latency of a step: with the layer's constants in registers, one
   block of code per step, the longest-lived simulations first and merged
   last packets, 200 simulations of the benchmark's range took 180 ms
   instead of 268, 32 smaller ones 101 instead of 138. */
template <bool RMAX>
static __device__ __forceinline__ bool batch_step(const McgbBatchConfig &cfg, const BatchPrep *prep,
                                                  const BatchLayer &c, BatchPacket &s, Rng &rng,
                                                  float rmax2, uint64_t *tally) {
    const float u = rng.next();
    Rng srng = rng;
    f3 sdir = s.dir;
    float az, ct = pf_sample<MCGB_PF_HG>(c.pf0, make_float4(c.pf1.x, c.pf1.y, 0.0f, 0.0f), nullptr, srng,
                                         &az, sdir);
    scatter_direction<true>(sdir, ct, az);
    float step = sample_step(u, c.factor);
    step = fminf(step, FLT_MAX);
    const float z = s.pos.z + step * s.dir.z;
    bool done = false;
    int layer = 1, next = 1;
    if (z < 0.0f || z >= c.thickness) {
        if (z < 0.0f) {
            --next;
            if (fabsf(s.dir.z) != 0.0f) step = mc_div(0.0f - s.pos.z, s.dir.z);
        }
        if (s.pos.z + step * s.dir.z >= c.thickness) {
            ++next;
            if (fabsf(s.dir.z) != 0.0f) step = mc_div(c.thickness - s.pos.z, s.dir.z);
        }
        s.pos.x = s.pos.x + s.dir.x * step;
        s.pos.y = s.pos.y + s.dir.y * step;
        s.pos.z = s.pos.z + s.dir.z * step;
        if (next > 1) s.pos.z = c.thickness;
        if (next < 1) s.pos.z = 0.0f;
        if (next != 1) {
            const BatchPrep &p = prep[s.rec];
            mcml_boundary(p.L, layer, next, s.dir, rng);
            if (layer != 1) {
                if (layer == 0) {
                    /* Radial detector, xopto/mcml/mcdetector/radial.py:117-150 */
                    float r = mc_sqrt(s.pos.x * s.pos.x + s.pos.y * s.pos.y);
                    int idx = clip_i(cvt_int(r * cfg.inv_dr), 0, (int)cfg.num_bins - 1);
                    uint32_t wi = weight_to_u32(s.w, 1.0f);
                    if (wi > 0) accu_add(tally, (uint64_t)p.sim * cfg.num_bins + idx, wi);
                }
                done = true;
            }
        }
    } else {
        s.pos.x = s.pos.x + s.dir.x * step;
        s.pos.y = s.pos.y + s.dir.y * step;
        s.pos.z = s.pos.z + s.dir.z * step;
    }
    if (next == 1) {
        float deposit = s.w * c.absorb;
        s.w -= deposit;
        rng = srng;
        s.dir = sdir;
        if (s.w < 1e-4f) {
            if (rng.next() > 0.1f) done = true;
            else s.w = mc_div(s.w, 0.1f);
        }
    }
    if (RMAX && dot3(s.pos, s.pos) > rmax2) done = true;
    return done;
}

template <bool RMAX>
__global__ void __launch_bounds__(256)
batched_kernel(const McgbBatchConfig cfg, const uint32_t *__restrict__ mult,
               const uint64_t *__restrict__ prefix, const BatchPrep *__restrict__ prep,
               unsigned long long *queue, uint64_t *tally, uint64_t *counters, uint64_t deadline_ns) {
    __shared__ BatchExchange share;
    ws_init(share);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t S = cfg.num_sims;
    const uint64_t total = prefix[S];
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const bool takes = ws_takes(share, total, 0u, warps);
    const float rmax2 = cfg.rmax * cfg.rmax;
    const uint64_t t_deadline = globaltimer_ns() + deadline_ns;

    uint64_t item_next = 0, item_end = 0;   /* warp-uniform */
    bool more = true;                         /* warp-uniform */
    bool active = false;
    BatchPacket s;
    s.rec = 0;
    BatchLayer c;
    Rng rng{0ull, 0u};
    uint64_t steps = 0, packets = 0;
    uint32_t iter = 0, status = 0;

    for (;;) {
        /* refill idle lanes with the next packets of the warp's item */
        uint32_t need = __ballot_sync(WS_FULL, takes && !active);
        while (need && more) {
            if (item_next >= item_end) {
                ws_fetch(queue, total, 0u, cfg.packets_per_item, warps, __popc(need), item_next, item_end);
                if (item_next >= total) {
                    more = false;
                    break;
                }
            }
            uint32_t avail = (uint32_t)min(item_end - item_next, (uint64_t)32);
            uint32_t rank = __popc(need & ((1u << lane) - 1u));
            bool mine = ((need >> lane) & 1u) && rank < avail;
            if (mine) {
                uint64_t g = item_next + rank;
                /* largest s with prefix[s] <= g (skips empty simulations) */
                uint32_t lo = 0, hi = S;
                while (lo < hi) {
                    uint32_t mid = (lo + hi + 1u) >> 1;
                    if (prefix[mid] <= g) lo = mid;
                    else hi = mid - 1u;
                }
                s.rec = lo;
                const BatchPrep &p = prep[lo];
                uint64_t x;
                uint32_t a;
                br_packet_stream(cfg.seed, p.sim, g - prefix[lo], mult, cfg.num_multipliers, &x, &a);
                rng = Rng{x, a};
                c.load(p);
                /* Line source at normal incidence (xopto/mcml/mcsource/line.py:95-108) */
                s.w = 1.0f - p.reflectance;
                s.pos = f3{0.0f, 0.0f, 0.0f};
                s.dir = f3{0.0f, 0.0f, 1.0f};
                active = true;
            }
            uint32_t taken = __ballot_sync(WS_FULL, mine);
            item_next += __popc(taken);
            need &= ~taken;
        }
        if (!more) {
            const bool had = active;
            if (!ws_share(share, active, [&](auto &io) { batch_state(io, s, rng); })) break;
            if (active && !had) c.load(prep[s.rec]);
        }

        /* sixteen steps between refills, two step bodies per loop
           iteration: the refill's ballots and queue reads cost more than the
           idle lanes of a packet that ends early (+2.4 % against eight steps
           without unrolling).  Once the queue is empty 64: the longest
           packets are then a serial chain, which each try at the exchange
           interrupts (32 simulations 101 -> 91 ms) */
        uint32_t taken = 0;
        const uint32_t count = more ? 16u : 64u;
#pragma unroll 2
        for (uint32_t k = 0; k < count; ++k) {
            if (active) {
                ++taken;
                if (batch_step<RMAX>(cfg, prep, c, s, rng, rmax2, tally)) {
                    active = false;
                    ++packets;
                }
            }
        }
        steps += taken;
        iter += count;
        if (iter >= 1024u) {
            iter = 0;
            uint32_t stop = 0;
            if (lane == 0) {
                if (globaltimer_ns() > t_deadline) stop = MCGB_STATUS_TIMEOUT;
                else if (*(volatile uint64_t *)(counters + MCGB_CNT_ABORT)) stop = MCGB_STATUS_ABORTED;
            }
            stop = __shfl_sync(WS_FULL, stop, 0);
            if (stop) {
                status |= stop;
                ws_leave(share);
                break;
            }
        }
    }
    warp_finish(counters, steps, packets, status);
}

}  // namespace MCGB_NS
