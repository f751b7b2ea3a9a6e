// trace_kernels.cu -- persistent traversal kernels of the wavefront.
//
// One lane traces one ray.  Warps are persistent (the grid is a fixed multiple
// of the SM count and the number of rays is read on the device, which keeps the
// frame capturable in a CUDA graph).  Each warp takes chunks of rays from
// a global counter (Knobs) and, between traversal steps, hands a new ray to every lane
// whose ray has finished, so lanes do not idle until the warp's longest ray ends
// (Aila & Laine, HPG 2009, persistent threads with ray replacement).  The short
// traversal stack of every lane lives in shared memory (STACK_SH entries) with a
// local spill.
#include "snk_frame.h"
#include "snk_trace.cuh"
#include "snk_shade.cuh"

namespace snk {
namespace {

constexpr int TBLK = 128;

// Launch knobs of a queue of n rays.  At each fetch a warp takes a quarter
// of its share of the rays that are left: the knob's 64 while the queue is long (few
// atomics, neighbouring rays in one warp), less towards its end, so that the warps finish
// together; but at least four times its share of the whole queue up to a warp's 32
// rays (a small queue fills warps with neighbours), and one ray per warp when there
// are fewer rays than that.  With always 64 the queue's end, and any queue of
// fewer rays than 64 per resident warp (233,472), left most warps without work: 64
// rays traced by one warp took 0.54 ms, one warp each 0.08 ms; a 65,536-path room frame
// 0.407 and 0.312 ms, the small 8-view terrain batch 2.37 and 1.60 ms, 1080p 2.19
// and 2.12 ms.  (Caps on the lanes that take rays, and asking for the next chunk
// ahead, gained nothing.)
constexpr uint32_t CHUNK_MAX = 64, CHUNK_MIN = 32;

struct Knobs {
    uint32_t chunk, chunk_min;
    bool coop;        // a warp's last rays may get eight lanes each
    uint32_t few;     // rays per warp of a queue of at most COOP_RAYS rays per resident warp, else 0
    float share;      // chunk per ray left
    int refill_idle;
    uint32_t prim_bias;
    __device__ __forceinline__ Knobs(const TraceTuning& t, uint32_t n, uint32_t bias = 3u)
        : chunk(t.chunk ? t.chunk : CHUNK_MAX), coop(t.default_limits != 0u), share(0.25f / (float)t.warps),
          refill_idle(t.refill_idle ? (int)t.refill_idle : 4), prim_bias(t.prim_bias ? t.prim_bias : bias) {
        const uint32_t c = (uint32_t)((float)n * (16.0f * share));
        chunk_min = min(max(c, 1u), min(CHUNK_MIN, chunk));
        few = coop && n <= (uint32_t)COOP_RAYS * t.warps ? max((n + t.warps - 1u) / t.warps, 1u) : 0u;
    }
    // eight lanes per ray from the start: a warp takes `few` rays at a time
    __device__ __forceinline__ void take_few() { chunk = chunk_min = few; }
    // the chunk to take when at most `left` rays are left
    __device__ __forceinline__ uint32_t next_chunk(uint32_t left) const {
        return min(max((uint32_t)((float)left * share), chunk_min), chunk);
    }
};

// One warp-voted traversal step: every active lane first pops until it has work
// (or finishes); then the warp runs either a node step in the lanes that have an
// internal child pending or a primitive step in the lanes that have a primitive
// pending, whichever more lanes want.  Returns true for a lane whose ray finished.
template <class TV>
__device__ __forceinline__ bool warp_step(TV& tv, bool active, const SceneDev& S, TraceCounters* ctr,
                                          uint32_t prim_bias) {
    if (active) tv.settle();
    const unsigned want_prim = __ballot_sync(0xFFFFFFFFu, active && tv.has_prim());   // (a finished ray has neither)
    const unsigned want_node = __ballot_sync(0xFFFFFFFFu, active && tv.has_node());
    const bool prims = 4u * (uint32_t)__popc(want_prim) >= prim_bias * (uint32_t)__popc(want_node);
    const uint32_t lane = threadIdx.x & 31u;
    if (prims) {
        if ((want_prim >> lane) & 1u) tv.prim_step(S, ctr);
    } else {
        if ((want_node >> lane) & 1u) tv.node_step(S, ctr);
    }
    return active && tv.done;
}

template <bool COUNT>
__device__ __forceinline__ void flush_counts(const TraceCounters& c, unsigned long long* out) {
    if (!COUNT || !out) return;
    unsigned long long a = c.nodes, b = c.tris;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xFFFFFFFFu, a, o);
        b += __shfl_down_sync(0xFFFFFFFFu, b, o);
    }
    if ((threadIdx.x & 31u) == 0) { atomicAdd(&out[0], a); atomicAdd(&out[1], b); }
}

// Warp-uniform source of ray indices: a local chunk refilled from `work`.
struct RayFeed {
    uint32_t next, end;
    bool exhausted;
    __device__ __forceinline__ void init() { next = 0; end = 0; exhausted = false; }
    // Assigns new indices to the idle lanes (mask `idle`); returns this lane's index
    // or INVALID.  Must be called by the whole warp.
    __device__ __forceinline__ uint32_t refill(unsigned idle, uint32_t lane, uint32_t* work, uint32_t n,
                                               const Knobs& kn) {
        if (next >= end && !exhausted) {
            uint32_t b = 0;
            const uint32_t chunk = kn.next_chunk(n - end);
            if (lane == 0) b = atomicAdd(work, chunk);
            b = __shfl_sync(0xFFFFFFFFu, b, 0);
            if (b >= n) {
                exhausted = true;
            } else {
                next = b;
                end = min(b + chunk, n);
            }
        }
        uint32_t mine = INVALID;
        if (next < end) {
            uint32_t i = next + __popc(idle & ((1u << lane) - 1u));
            if (((idle >> lane) & 1u) && i < end) mine = i;
            next = min(next + (uint32_t)__popc(idle), end);
        }
        return mine;
    }
    __device__ __forceinline__ bool done() const { return exhausted && next >= end; }
};

// Traces a queue: `refill(idle)` gives the lanes of the mask their next entries (INVALID:
// none), `done()` tells that there are no more; start(tv, entry) sets a ray up and
// returns the index its result goes to, emit(tv, index) writes the result of a finished
// ray.  COOP: a warp's last COOP_RAYS rays get eight lanes each (coop_trace) once one of
// them has taken COOP_STEPS steps: such a ray has a long way behind it and likely more to
// go, and the queue's end waits for it (short rays, as in a closed room, finish sooner
// where they are: a 65,536-path room frame 304 us, 328 with all last rays moved).  So do
// all rays of a queue that gives the resident warps no more than COOP_RAYS each.  (Not with
// limits of the caller's: eight lanes take a leaf's triangles in one step and keep fewer
// entries, so that it would depend on a ray's queue whether a limit is reported.)  The
// 480x270 terrain batch took 1.43 instead of 1.55 ms so, a 480x270 sphere-field frame 0.54
// and 0.58, a 1080p frame 2.005 and 2.037, 10,000 rays 112 and 129 us, 64 rays 73 and 83 us.
constexpr uint32_t COOP_STEPS = 48;

template <bool COOP, class TV, class Refill, class Done, class Start, class Emit>
__device__ __forceinline__ void trace_queue(const SceneDev& S, const Knobs& kn, uint2* sh_stack, TraceCounters* ctr,
                                            Refill&& refill, Done&& done, Start&& start, Emit&& emit) {
    __shared__ CoopSlot coop_slots[COOP ? TBLK / 32 : 1][COOP_RAYS];
    uint2 spill[STACK_MAX - STACK_SH];
    auto rank = [](unsigned mask) { return (uint32_t)__popc(mask & ((1u << (threadIdx.x & 31u)) - 1u)); };
    auto finish_few = [&](uint32_t k) {   // the k rays in the warp's slots
        if constexpr (COOP) {
            CoopSlot* slots = coop_slots[threadIdx.x >> 5];
            coop_trace<!TV::ORD>(slots, k, S, sh_stack, spill, TBLK);
            const uint32_t lane = threadIdx.x & 31u;
            if (lane < k) {
                TraceResult r;
                ray_result(slots[lane], S, r);
                emit(r, slots[lane].ri);
            }
            __syncwarp();
        }
    };
    TV tv;
    if (COOP && kn.few) {
        do {
            const uint32_t i = refill((1u << kn.few) - 1u);
            const unsigned act = __ballot_sync(0xFFFFFFFFu, i != INVALID);
            if (i != INVALID) {
                const uint32_t ri = start(tv, i, spill);
                coop_save(coop_slots[threadIdx.x >> 5][rank(act)], tv, ri);
            }
            if (act) finish_few((uint32_t)__popc(act));
        } while (!done());
        return;
    }
    bool active = false;
    uint32_t ri = 0;
    for (;;) {
        unsigned act = __ballot_sync(0xFFFFFFFFu, active);
        if (__popc(~act) >= kn.refill_idle) {
            if (!done()) {
                const uint32_t i = refill(~act);
                if (i != INVALID) {
                    ri = start(tv, i, spill);
                    active = true;
                }
                act = __ballot_sync(0xFFFFFFFFu, active);
                if (act == 0) continue;
            } else if (act == 0) {
                break;
            } else if (COOP && kn.coop && __popc(act) <= COOP_RAYS &&
                       __any_sync(0xFFFFFFFFu, active && tv.steps >= COOP_STEPS)) {
                if (active) coop_save(coop_slots[threadIdx.x >> 5][rank(act)], tv, ri);
                finish_few((uint32_t)__popc(act));
                break;
            }
        }
        if (warp_step(tv, active, S, ctr, kn.prim_bias)) {
            TraceResult r;
            tv.finish(S, r);
            emit(r, ri);
            active = false;
        }
    }
}

__device__ __forceinline__ void store_hit(HitDev* dst, const TraceResult& r) {
    HitDev h;
    h.t = r.t; h.inst = r.inst; h.prim = r.prim; h.u = r.u; h.v = r.v; h.flags = r.hit ? 1u : 0u;
    uint2* d = reinterpret_cast<uint2*>(dst);
    const uint2* s = reinterpret_cast<const uint2*>(&h);
    d[0] = s[0]; d[1] = s[1]; d[2] = s[2];
}

// closest hit of the rays queued for segment d
template <bool COUNT, int MINB, bool SINGLE>
__global__ void __launch_bounds__(TBLK, MINB) k_trace_closest(const __grid_constant__ FrameParams F, uint32_t d) {
    constexpr bool COOP = SINGLE && !COUNT;
    using TV = Traverser<false, COUNT, SINGLE>;
    __shared__ uint2 sh_stack[TRACE_SH_ROWS * TBLK];
    const uint32_t n = F.counters[CNT_QUEUE + d];
    Knobs kn(F.tune, n);
    if (COOP && kn.few) kn.take_few();
    const float4* rays = F.rays[d & 1u];
    uint32_t* work = &F.counters[CNT_WORK_TRACE + d];
    const uint32_t lane = threadIdx.x & 31u;
    TraceCounters ctr{0ull, 0ull};
    RayFeed feed;
    feed.init();
    trace_queue<COOP, TV>(
        F.S, kn, sh_stack, &ctr, [&](unsigned idle) { return feed.refill(idle, lane, work, n, kn); },
        [&] { return feed.done(); },
        [&](TV& tv, uint32_t i, uint2* spill) {
            const float4 a = __ldg(rays + 2ull * i), b = __ldg(rays + 2ull * i + 1);
            tv.init(F.S, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), a.w, b.w, sh_stack, spill, threadIdx.x, TBLK);
            return i;
        },
        [&](const TraceResult& r, uint32_t ri) {
            if (r.hit) store_hit(F.hits + ri, r);
            else F.hits[ri].flags = 0u;   // (all that is read of a miss)
        });
    flush_counts<COUNT>(ctr, F.trav_counters);
}

// closest hits of segment d's rays in warp packets of 32 consecutive queue entries
// (the camera segment: the 32 pixels of one 8 x 4 tile per warp)
template <int MINB>
__global__ void __launch_bounds__(TBLK, MINB) k_trace_packet(FrameParams F, uint32_t d) {
    __shared__ uint4 sh_pstack[(TBLK / 32) * PSTACK];
    __shared__ uint2 sh_world[5 * TBLK];
    const uint32_t n = F.counters[CNT_QUEUE + d];
    const float4* rays = F.rays[d & 1u];
    uint32_t* work = &F.counters[CNT_WORK_TRACE + d];
    const uint32_t lane = threadIdx.x & 31u;
    uint4* stack = sh_pstack + (threadIdx.x >> 5) * PSTACK;
    for (;;) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(work, 32u);
        b = __shfl_sync(0xFFFFFFFFu, b, 0);
        if (b >= n) break;
        const uint32_t i = b + lane;
        const bool active = i < n;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = a;
        if (active) { a = __ldg(rays + 2ull * i); c = __ldg(rays + 2ull * i + 1); }
        PacketTraverser<false, TBLK> tv;
        tv.init(F.S, v3(a.x, a.y, a.z), v3(c.x, c.y, c.z), a.w, c.w, active, stack, sh_world + threadIdx.x);
        tv.run(F.S);
        TraceResult r;
        tv.finish(F.S, r);
        if (active && r.hit) store_hit(F.hits + i, r);
        if (active && !r.hit) F.hits[i].flags = 0u;
    }
}

// shadow rays of segment d: the compacted queue's n0 directional-light rays (origins
// only: the eight-view terrain batch 36.38 -> 36.26 ms), then its n1 local-light rays
// (from ray n_paths on).  A ray's origin w holds its
// contribution entry (shadow_entry); the visibility goes to that entry's byte
// (shadow_vis), and k_accum_shadow adds the visible contributions in entry order
// (the same order as the CPU oracle, so sums are bit-identical).
template <bool COUNT, int MINB, bool SINGLE>
__global__ void __launch_bounds__(TBLK, MINB) k_trace_shadow(const __grid_constant__ FrameParams F, uint32_t d) {
    constexpr bool COOP = SINGLE && !COUNT;
    using TV = Traverser<true, COUNT, SINGLE>;
    __shared__ uint2 sh_stack[TRACE_SH_ROWS * TBLK];
    const uint32_t n0 = F.counters[CNT_SHADOW_Q + 2 * d], n = n0 + F.counters[CNT_SHADOW_Q + 2 * d + 1];
    Knobs kn(F.tune_any, n);
    if (COOP && kn.few) kn.take_few();
    uint32_t* work = &F.counters[CNT_WORK_SHADOW + d];
    const uint32_t lane = threadIdx.x & 31u;
    TraceCounters ctr{0ull, 0ull};
    RayFeed feed;
    feed.init();
    trace_queue<COOP, TV>(
        F.S, kn, sh_stack, &ctr, [&](unsigned idle) { return feed.refill(idle, lane, work, n, kn); },
        [&] { return feed.done(); },
        [&](TV& tv, uint32_t j, uint2* spill) {
            const float* dl = F.S.dir_light.dir;
            float4 a, b = make_float4(dl[0], dl[1], dl[2], T_FAR);
            if (j < n0) {
                a = __ldg(F.shadow_rays + j);
            } else {
                const float4* sr = F.shadow_rays + 2 * ((size_t)F.n_paths + (j - n0));
                a = __ldg(sr);
                b = __ldg(sr + 1);
            }
            tv.init(F.S, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), SHADOW_TMIN, b.w, sh_stack, spill, threadIdx.x, TBLK);
            return __float_as_uint(a.w);
        },
        [&](const TraceResult& r, uint32_t ri) { shadow_vis(F)[ri] = r.hit ? 0u : 1u; });
    flush_counts<COUNT>(ctr, F.trav_counters ? F.trav_counters + 2 : nullptr);
}

// adds the visible shadow-ray contributions of segment d to the path radiance, which
// segment 0's (of every path) start; an emitter met by a camera ray is such a contribution.
// (The generation wrote a throughput of 1 and a radiance of 0 for every path and the
// first shading and shadow passes read them back, 64 bytes a path: a 1080p frame of
// the sphere field 1.921 ms, 1.899 so.)
__global__ void __launch_bounds__(256) k_accum_shadow(FrameParams F, uint32_t d) {
    const uint32_t n = F.counters[CNT_QUEUE + d];
    const uint32_t* pids = F.path_ids[d & 1u];
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
        const bool v0 = shadow_vis(F)[shadow_entry(F, i, 0)] != 0u, v1 = shadow_vis(F)[shadow_entry(F, i, 1)] != 0u;
        const bool add = v0 || v1;
        uint32_t p = 0;
        bool fin = false;   // (early resolve) the path ends in this segment
        if (F.early_resolve) {
            const uint32_t raw = pids[i];
            p = raw & 0x7FFFFFFFu;
            fin = (raw >> 31) != 0u;
        } else {
            if (!add && d) continue;
            p = pids[i];
        }
        if (!add && !fin && d) continue;
        float4 l = d ? F.L[p] : make_float4(0.0f, 0.0f, 0.0f, 0.0f), c0 = l, c1 = l;
        if (v0) c0 = F.shadow_contrib[shadow_entry(F, i, 0)];
        if (v1) c1 = F.shadow_contrib[shadow_entry(F, i, 1)];
        if (v0) l = make_float4(l.x + c0.x, l.y + c0.y, l.z + c0.z, 0.0f);
        if (v1) l = make_float4(l.x + c1.x, l.y + c1.y, l.z + c1.z, 0.0f);
        if (fin) {   // the pixel's outputs, as the resolve pass writes them for one sample
            const uint32_t vi = find_view(F.views, F.nviews, p);   // (one sample: path p is pixel p)
            const ViewDev& V = F.views[vi];
            const uint32_t o = p - V.pixel_offset;
            const float4 r = make_float4(l.x, l.y, l.z, 1.0f);
            if (V.radiance) V.radiance[o] = r;
            if (vi == 0 && frame_accumulate(F)) {
                double2 a0 = F.accum[2ull * o], a1 = F.accum[2ull * o + 1];
                a0.x += (double)r.x; a0.y += (double)r.y; a1.x += (double)r.z; a1.y += 1.0;
                F.accum[2ull * o] = a0;
                F.accum[2ull * o + 1] = a1;
            }
            continue;
        }
        F.L[p] = l;
        if (F.cache && p >= F.n_render) {   // radiance gathered at this vertex of a training path
            const uint32_t slot = (p - F.n_render) * TRAIN_V + (d < TRAIN_V - 1 ? d : TRAIN_V - 1);
            float4 v = F.train_L[slot];
            if (v0) v = make_float4(v.x + c0.x, v.y + c0.y, v.z + c0.z, 0.0f);
            if (v1) v = make_float4(v.x + c1.x, v.y + c1.y, v.z + c1.z, 0.0f);
            F.train_L[slot] = v;
        }
    }
}

// i / pixels and i % pixels (recip: 2^32 / pixels)
__device__ __forceinline__ uint32_t slot_of(uint32_t i, uint32_t pixels, uint32_t recip, uint32_t* pixel) {
    uint32_t k = __umulhi(i, recip), o = i - k * pixels;   // (that, or one less)
    if (o >= pixels) { o -= pixels; k++; }
    *pixel = o;
    return k;
}

// Ray feed over a queue with entries not in use (RestirQueue::counts): the warp takes 32 entries
// at a time from the work counter, keeps the real ones in a per-warp ring in
// shared memory and hands only those to its idle lanes, so an empty entry costs
// one load of its pixel's count instead of a lane's turn.
struct FilteredFeed {
    RayFeed raw;
    uint32_t head, cnt;   // the ring's pending entries (warp-uniform)
    __device__ __forceinline__ void init() { raw.init(); head = 0; cnt = 0; }
    __device__ __forceinline__ uint32_t refill(unsigned idle, uint32_t lane, uint32_t* work, uint32_t n, const Knobs& kn,
                                               const uint8_t* counts, uint32_t pixels, uint32_t recip,
                                               uint32_t* ring) {
        const uint32_t nidle = (uint32_t)__popc(idle), lt = (1u << lane) - 1u;
        while (cnt < nidle && !raw.done()) {   // (cnt < 32 here, so the ring of 64 never overflows)
            const uint32_t e = raw.refill(0xFFFFFFFFu, lane, work, n, kn);
            bool real = e != INVALID;
            if (real) {
                uint32_t o;
                const uint32_t k = slot_of(e, pixels, recip, &o);
                real = k < __ldg(counts + o);
            }
            const unsigned rm = __ballot_sync(0xFFFFFFFFu, real);
            if (real) ring[(head + cnt + (uint32_t)__popc(rm & lt)) & 63u] = e;
            cnt += (uint32_t)__popc(rm);
            __syncwarp();
        }
        uint32_t mine = INVALID;
        const uint32_t r = (uint32_t)__popc(idle & lt);
        if (((idle >> lane) & 1u) && r < cnt) mine = ring[(head + r) & 63u];
        const uint32_t take = nidle < cnt ? nidle : cnt;
        head = (head + take) & 63u;
        cnt -= take;
        __syncwarp();
        return mine;
    }
    __device__ __forceinline__ bool done() const { return raw.done() && cnt == 0; }
};

// Where the rest of a segment of length t starts whose first t - PL_SHORTER is free: one
// float below that, since a test takes neither of its ends and a hit at t - PL_SHORTER is in
// the whole segment (of a difference of 0 that makes a NaN, of a negative one a negative
// one: SHADOW_TMIN).
__device__ __forceinline__ float end_tmin(float t) {
    return fmaxf(SHADOW_TMIN, __uint_as_float(__float_as_uint(t - PL_SHORTER) - 1u));
}

// visibility of a queue of segments (RestirQueue): vis[i] = 1 when nothing is hit in (tmin,
// tmax), 0 when something is; entries not in use are skipped, vis[i] not written:
// the passes never read the result of a slot they did not record.  Origins are kept once
// per pixel and the number of slots in use as a byte instead of marks in the others: the
// recording passes are bound by the slots' bytes (two 1080p frames 14.19 -> 13.96 ms, and
// 13.98 -> 13.83).
// The ReSTIR passes queue their visibility rays here instead of tracing inline.  (No
// eight-lane end: these queues are long and their rays short, two 1080p ReSTIR frames
// took 17.38 ms with it and 17.02 without.)
template <int MINB, bool SINGLE>
__global__ void __launch_bounds__(TBLK, MINB) k_trace_visibility(const __grid_constant__ SceneDev S, const float4* __restrict__ rays,
                                                                 const float4* __restrict__ origin,
                                                                 const uint8_t* __restrict__ counts, uint32_t pixels,
                                                                 uint32_t recip, uint32_t n, uint8_t* vis,
                                                                 uint32_t* work, TraceTuning tune) {
    using TV = Traverser<true, false, SINGLE>;
    __shared__ uint2 sh_stack[TRACE_SH_ROWS * TBLK];
    __shared__ uint32_t ring[TBLK / 32][64];
    const Knobs kn(tune, n, 2u);   // (few triangles a ray: two ReSTIR frames 13.59 ms, 13.68 with 3, 13.62 with 1)
    const uint32_t lane = threadIdx.x & 31u;
    FilteredFeed feed;
    feed.init();
    trace_queue<false, TV>(
        S, kn, sh_stack, nullptr,
        [&](unsigned idle) { return feed.refill(idle, lane, work, n, kn, counts, pixels, recip, ring[threadIdx.x >> 5]); },
        [&] { return feed.done(); },
        [&](TV& tv, uint32_t i, uint2* spill) {
            uint32_t o;
            slot_of(i, pixels, recip, &o);
            const float4 b = __ldg(rays + i), a = __ldg(origin + o);
            const float t = fabsf(b.w);
            tv.init(S, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), b.w < 0.0f ? end_tmin(t) : SHADOW_TMIN, t, sh_stack, spill,
                    threadIdx.x, TBLK);
            return i;
        },
        [&](const TraceResult& r, uint32_t ri) { vis[ri] = r.hit ? 0u : 1u; });
}

// trace of an array of rays: snk_pt_trace_rays, and the rays of the particle and contact queries
template <bool ANY, bool SINGLE>
__global__ void __launch_bounds__(TBLK, 6) k_trace_rays(const __grid_constant__ SceneDev S, const float4* __restrict__ rays, uint32_t n,
                                                     HitDev* hits, uint32_t* work, TraceTuning tune) {
    using TV = Traverser<ANY, false, SINGLE>;
    __shared__ uint2 sh_stack[TRACE_SH_ROWS * TBLK];
    Knobs kn(tune, n);
    if (SINGLE && kn.few) kn.take_few();
    const uint32_t lane = threadIdx.x & 31u;
    RayFeed feed;
    feed.init();
    trace_queue<SINGLE, TV>(
        S, kn, sh_stack, nullptr, [&](unsigned idle) { return feed.refill(idle, lane, work, n, kn); },
        [&] { return feed.done(); },
        [&](TV& tv, uint32_t i, uint2* spill) {
            const float4 a = __ldg(rays + 2ull * i), b = __ldg(rays + 2ull * i + 1);
            tv.init(S, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), a.w, b.w, sh_stack, spill, threadIdx.x, TBLK);
            return i;
        },
        [&](TraceResult r, uint32_t ri) {
            if (ANY) {
                r.t = r.hit ? 1.0f : -1.0f; r.inst = INVALID; r.prim = INVALID; r.u = 0.0f; r.v = 0.0f;
            }
            store_hit(hits + ri, r);
        });
}

}  // namespace

// register budget variants: 0 -> at most 85 registers (6 blocks of 128 per SM),
// 1 -> 64 registers (8 blocks), 2 -> unconstrained (4 blocks); each in the
// single-primitive-leaf form when the scene's trees allow it
template <bool COUNT, bool SINGLE>
void launch_closest_variant(const FrameParams& F, uint32_t depth, int grid, cudaStream_t s) {
    if (F.tune.variant == 1) k_trace_closest<COUNT, 8, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
    else if (F.tune.variant == 2) k_trace_closest<COUNT, 4, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
    else k_trace_closest<COUNT, 6, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
}
template <bool COUNT, bool SINGLE>
void launch_shadow_variant(const FrameParams& F, uint32_t depth, int grid, cudaStream_t s) {
    if (F.tune_any.variant == 1) k_trace_shadow<COUNT, 8, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
    else if (F.tune_any.variant == 2) k_trace_shadow<COUNT, 4, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
    else k_trace_shadow<COUNT, 6, SINGLE><<<grid, TBLK, 0, s>>>(F, depth);
}

cudaError_t launch_trace_closest(const FrameParams& F, uint32_t depth, int grid, bool count, cudaStream_t s) {
    const bool single = F.S.single_leaf != 0u;
    // camera rays (segment 0) in warp packets when the frame allows them
    // (FrameParams::packet_primary; a counting launch always traces ray by ray)
    if (depth == 0 && F.packet_primary && !count) {
        k_trace_packet<6><<<grid, TBLK, 0, s>>>(F, depth);
        return cudaGetLastError();
    }
    if (count) single ? launch_closest_variant<true, true>(F, depth, grid, s) : launch_closest_variant<true, false>(F, depth, grid, s);
    else single ? launch_closest_variant<false, true>(F, depth, grid, s) : launch_closest_variant<false, false>(F, depth, grid, s);
    return cudaGetLastError();
}

cudaError_t launch_trace_shadow(const FrameParams& F, uint32_t depth, int grid, bool count, cudaStream_t s) {
    const bool single = F.S.single_leaf != 0u;
    if (count) single ? launch_shadow_variant<true, true>(F, depth, grid, s) : launch_shadow_variant<true, false>(F, depth, grid, s);
    else single ? launch_shadow_variant<false, true>(F, depth, grid, s) : launch_shadow_variant<false, false>(F, depth, grid, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_accum_shadow<<<grid / 2 > 0 ? grid / 2 : 1, 256, 0, s>>>(F, depth);
    return cudaGetLastError();
}

cudaError_t launch_trace_visibility(const SceneDev& S, const float4* rays, const float4* origin, const uint8_t* counts,
                                    uint32_t pixels, uint32_t n, uint8_t* vis, uint32_t* work, int grid,
                                    const TraceTuning& tune, cudaStream_t s) {
    const uint32_t recip = pixels > 1u ? (uint32_t)(0x100000000ull / pixels) : 0xFFFFFFFFu;
    if (S.single_leaf) {
        if (tune.variant == 1) k_trace_visibility<8, true><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
        else if (tune.variant == 2) k_trace_visibility<4, true><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
        else k_trace_visibility<6, true><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
    } else {
        if (tune.variant == 1) k_trace_visibility<8, false><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
        else if (tune.variant == 2) k_trace_visibility<4, false><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
        else k_trace_visibility<6, false><<<grid, TBLK, 0, s>>>(S, rays, origin, counts, pixels, recip, n, vis, work, tune);
    }
    return cudaGetLastError();
}

cudaError_t launch_trace_rays(const SceneDev& S, const float4* rays, uint32_t n, HitDev* hits, bool any,
                              uint32_t* work, int grid, const TraceTuning& tune, cudaStream_t s) {
    if (S.single_leaf) {
        if (any) k_trace_rays<true, true><<<grid, TBLK, 0, s>>>(S, rays, n, hits, work, tune);
        else k_trace_rays<false, true><<<grid, TBLK, 0, s>>>(S, rays, n, hits, work, tune);
    } else {
        if (any) k_trace_rays<true, false><<<grid, TBLK, 0, s>>>(S, rays, n, hits, work, tune);
        else k_trace_rays<false, false><<<grid, TBLK, 0, s>>>(S, rays, n, hits, work, tune);
    }
    return cudaGetLastError();
}

}  // namespace snk
