// Device building blocks shared by the wavefront renderers (path tracer and
// density-grid medium): warp-aggregated queue slots and the persistent
// traversal loop over a ray queue.
#pragma once

#include "dev_common.cuh"
#include "trace.cuh"

namespace cupbr_b200 {

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Loads of wavefront state (queues, hits, radiance, counters).  NC = true:
// the read-only path (__ldg), for stage kernels, which never read what they
// themselves write.  NC = false: cached in L2 only (__ldcg), for the
// persistent batch kernel, whose stages read what other blocks of the same
// launch wrote before a grid barrier (an L1 or read-only cache line from an
// earlier stage could be stale).
template <bool NC, typename T>
__device__ __forceinline__ T qload(const T* p) {
    return NC ? __ldg(p) : __ldcg(p);
}

// Warp-aggregated slot allocation for the lanes with `want` set.
__device__ __forceinline__ uint32_t claim_slot(bool want, uint32_t* counter) {
    const unsigned full = 0xffffffffu;
    unsigned mask = __ballot_sync(full, want);
    if (mask == 0u) return 0u;
    int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
    base = __shfl_sync(full, base, leader);
    return base + (uint32_t)__popc(mask & ((1u << lane_id()) - 1u));
}

// Traversal stack of a persistent lane: the first LEVELS entries in shared
// memory, row by row over the block's threads (conflict free whatever the
// lanes' depths; in local memory lanes at different depths touch a line
// each), the rest in local memory.  Occlusion rays store references only.
// 12 and 16 levels take 96 and 64 KB of an SM at 8 blocks of 128 threads;
// with 8 the 1080p terrain took 46.1 ms instead of 45.4, with 6 47.4.
template <bool ANY, int THREADS>
struct LaneStack {
    static constexpr int LEVELS = ANY ? 16 : 12;
    static constexpr int ROW = THREADS * (ANY ? 4 : 8);  // bytes from one row to the next
    static constexpr int NEAR = LEVELS * ROW;
    static constexpr int FULL = CUPBR_STACK_SIZE * ROW;
    char* base;  // this thread's entry of row 0
    int sp;      // depth * ROW
    int32_t far_ref[CUPBR_STACK_SIZE - LEVELS];
    int32_t far_key[ANY ? 1 : CUPBR_STACK_SIZE - LEVELS];
    __device__ __forceinline__ LaneStack(char* s_stack) : base(s_stack + threadIdx.x * (ANY ? 4 : 8)), sp(0) {}
    __device__ __forceinline__ void clear() { sp = 0; }
    __device__ __forceinline__ bool empty() const { return sp == 0; }
    __device__ __forceinline__ void put(int at, int32_t key, int32_t ref) {
        if (ANY) *reinterpret_cast<int32_t*>(base + at) = ref;
        else *reinterpret_cast<int2*>(base + at) = make_int2(key, ref);
    }
    // room for three more entries in shared memory: put() them and raise sp
    __device__ __forceinline__ bool near3() const { return sp <= NEAR - 3 * ROW; }
    __device__ __forceinline__ void push(int32_t key, int32_t ref, bool& overflow) {
        if (sp < NEAR) {
            put(sp, key, ref);
        } else if (sp < FULL) {
            far_ref[(sp - NEAR) / ROW] = ref;
            if (!ANY) far_key[(sp - NEAR) / ROW] = key;
        } else {
            overflow = true;
            return;
        }
        sp += ROW;
    }
    __device__ __forceinline__ int2 pop() {
        sp -= ROW;
        if (sp < NEAR) {
            if (ANY) return make_int2(0, *reinterpret_cast<const int32_t*>(base + sp));
            return *reinterpret_cast<const int2*>(base + sp);
        }
        return make_int2(ANY ? 0 : far_key[(sp - NEAR) / ROW], far_ref[(sp - NEAR) / ROW]);
    }
};
template <int THREADS>
constexpr int TRACE_STACK_BYTES = LaneStack<false, THREADS>::NEAR;  // occlusion rays take 2/3 of it

// Resumes the next stack entry that can still hold a counted hit.
template <bool ANY, typename Stack>
__device__ __forceinline__ void trav_pop(TravState& s, Stack& st) {
    const int32_t limit = key_limit(s.t_best);
    for (;;) {
        if (st.empty()) { s.cur = TRAV_IDLE; return; }
        const int2 e = st.pop();
        if (ANY || e.x <= limit) { s.cur = e.y; return; }
    }
}

// Asks L2 for the bytes [p, p + bytes) that the block reads in its next chunk
// (p 16-byte aligned): the threads take a 128-byte line each.  The stage
// kernels read queues that the traversal wrote through to DRAM, at the head of
// a chain of dependent loads.
__device__ __forceinline__ void prefetch_block(const void* p, uint32_t bytes) {
    const uint32_t at = threadIdx.x * 128u;
    if (at < bytes)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(static_cast<const char*>(p) + at)));
}

// Queue slots for a block: lanes with want[k] set get consecutive slots of
// queue k, one atomicAdd per block and queue.  Every thread of the block calls
// it together.  The stage kernels push an entry or two per ray into two or
// three queues, and the additions to one counter complete one after the other
// (about 1.3 per ns on a B200): one per warp kept a shading stage at 0.2 ms
// per 4M rays whatever else it did.
template <int QUEUES, int WARPS>
struct BlockClaim {
    uint32_t count[QUEUES][WARPS];  // per warp, then each warp's first slot
    __device__ __forceinline__ void operator()(const bool (&want)[QUEUES], uint32_t* const (&counter)[QUEUES],
                                               uint32_t (&slot)[QUEUES]) {
        static_assert(QUEUES <= WARPS, "warp k adds up queue k");
        const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
        unsigned mask[QUEUES];
#pragma unroll
        for (int k = 0; k < QUEUES; ++k) {
            mask[k] = __ballot_sync(0xffffffffu, want[k]);
            if (lane == 0) count[k][wid] = (uint32_t)__popc(mask[k]);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < QUEUES; ++k) {
            if ((int)wid != k) continue;
            const uint32_t n = lane < WARPS ? count[k][lane] : 0u;
            uint32_t before = n;  // inclusive prefix over the warps
#pragma unroll
            for (int o = 1; o < WARPS; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
                if ((int)lane >= o) before += v;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, before, WARPS - 1);
            uint32_t base = 0;
            if (lane == 0 && total) base = atomicAdd(counter[k], total);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (lane < WARPS) count[k][lane] = base + before - n;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < QUEUES; ++k) slot[k] = count[k][wid] + (uint32_t)__popc(mask[k] & ((1u << lane) - 1u));
    }
};

constexpr int TRACE_NODE_STEPS = 3;
constexpr int TRACE_REFILL = 12;

// Queue entries a warp claims at once: a third of its share of what is left
// of the queue, 32 to 128.  Large claims spare the one counter (32 at a time
// doubled the shadow stage of a scene of 20 primitives), small ones keep the
// warps' last rays even (128 to the end: 1080p terrain +1 %, 512: +8 %).
__device__ __forceinline__ uint32_t trace_chunk(uint32_t count, uint32_t end, uint32_t warps) {
    const uint32_t left = count - min(end, count);
    return max(32u, min(128u, (left / (3u * warps)) & ~31u));
}

// A warp's part of a queue: entries [next, end) in hand, the first ones by the
// warp's number, later ones claimed from the counter (which counts from
// first_end on).  A queue of at most 32 entries per warp is dealt out whole, a
// few lanes to each warp: its warps then diverge less, and no counter is
// touched (its additions complete one after the other, 0.8 ns each: 4 us for
// the warps of a grid).  Four ragged 1273 x 717 frames in flight 6.6 -> 6.0 ms.
// Where frames overlap, other frames' warps fill the lanes that this leaves
// empty only as warps of their own: there a warp takes `least` = 32 (pipelined
// frames of the Cornell box, us each, 400 x 300 128 with least = 4, 99 with 32;
// 480 x 270 120 / 96; 640 x 360 148 / 119; a scene of 40 objects of all
// materials 99 / 101, 98 / 100, 114 / 113).
// Packets stay with 32 rays a claim: neighbouring packets then run at the same
// time (960 x 540 terrain 363 us, 556 with this deal).
struct TraceShare {
    uint32_t next, end;
    const uint32_t* first_end;  // in shared memory: read when a warp has used up what it holds
    static constexpr uint32_t DRY = 0xffffffffu;
    static __device__ __forceinline__ uint32_t warps() { return gridDim.x * (blockDim.x >> 5); }
    // every thread of the block calls it
    __device__ __forceinline__ TraceShare(uint32_t count, uint32_t least, uint32_t* s_first_end) {
        const uint32_t share = (count + warps() - 1u) / warps();
        const uint32_t first = share <= 32u ? max(share, least) : trace_chunk(count, 0u, warps());
        if (threadIdx.x == 0) *s_first_end = first * warps();
        __syncthreads();
        first_end = s_first_end;
        next = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * first;
        end = next + first;
    }
    __device__ __forceinline__ bool more(uint32_t count) const {
        if (next < end) return next < count;
        return next != DRY && *first_end < count;
    }
    // Entries for the n idle lanes of a warp (all lanes call it while there is
    // more): the index for the lane of rank r, not below count when there is
    // none for it.
    __device__ __forceinline__ uint32_t take(uint32_t count, uint32_t n, uint32_t r, uint32_t* fetch) {
        const uint32_t have = end - next;
        if (n <= have) {
            next += n;
            return next - n + r;
        }
        const uint32_t base = *first_end;
        if (base >= count) {  // the whole queue was dealt out
            const uint32_t i = r < have ? next + r : DRY;
            next = end = DRY;
            return i;
        }
        const uint32_t chunk = trace_chunk(count, max(end, base), warps());
        uint32_t fresh = 0;
        if (lane_id() == 0) fresh = atomicAdd(fetch, chunk);
        fresh = base + __shfl_sync(0xffffffffu, fresh, 0);
        const uint32_t i = r < have ? next + r : fresh + (r - have);
        next = end = DRY;
        if (fresh < count) {
            next = fresh + (n - have);  // n <= 32 <= chunk
            end = fresh + chunk;
        }
        return i;
    }
};

// Persistent traversal over a queue with per-lane dynamic fetch.  A warp's
// lanes walk the tree in rounds of at most TRACE_NODE_STEPS node visits and
// then one leaf: a bound on the visits, because a round that descends until
// every lane holds a leaf runs as long as its slowest lane.  Lanes whose
// ray is done wait until TRACE_REFILL of them (or the whole warp) can hand in
// their results and take the next rays together; the warp claims the queue in
// chunks, so a refill rarely waits for an atomic.  Entry i of the queue starts
// at q[stride * i]: (origin, ANY ? t_limit : -), (direction, -).  ANY = false:
// closest hit, ANY = true: occlusion up to t_limit.  done(i, state) runs once
// per ray.  s_stack: LaneStack<ANY, THREADS>::NEAR bytes of shared memory.
//
// Bound by issue slots and by the L1's load pipe (terrain, first bounce, B200:
// 60 % and 65 % busy).  Measured on the 1080p terrain / the 512^2 Cornell box
// (whole passes, one box): descent to a leaf by every lane and two such rounds
// between refills 52.0 / 11.32 ms; this 45.1 / 10.65 ms; 2 or 4 node visits
// 46.8 / 45.4 ms; a vote for the phase with more lanes before every step
// 47.1 / 12.2 ms (15 lanes busy, but the votes cost what they gain); one
// primitive per round instead of a leaf 50.7 / 13.4 ms; refills at 4 idle
// lanes 46.2 ms.
template <bool ANY, bool COUNT, int THREADS, bool NC = true, typename Done>
__device__ __forceinline__ void persistent_trace(const DeviceScene& S, const float4* __restrict__ q, uint32_t stride,
                                                 uint32_t count, uint32_t least, uint32_t* fetch, char* s_stack,
                                                 uint32_t* err_stack, uint64_t* stats, Done done) {
    const unsigned full = 0xffffffffu;
    const uint32_t lane = lane_id();
    // a well-formed tree visits every node at most once per ray, and a round
    // advances every lane that is on a ray
    const uint32_t guard = S.n_nodes + S.n_tris + S.n_spheres + S.n_quads + 64u;  // slots are below 2^28
    TravState s;
    s.cur = TRAV_IDLE;
    LaneStack<ANY, THREADS> st(s_stack);
    TraceCounters tc;
    __shared__ uint32_t s_first_end;
    TraceShare share(count, least, &s_first_end);
    bool overflow = false, have = false;
    uint32_t idx = 0;
    uint32_t steps = 0;
    for (;;) {
        const unsigned m_idle = __ballot_sync(full, s.cur == TRAV_IDLE);
        if (m_idle == full || (__popc(m_idle) >= TRACE_REFILL && share.more(count))) {
            // finished lanes hand in their results and take the next rays
            const bool idle = s.cur == TRAV_IDLE;
            if (idle && have) {
                have = false;
                done(idx, s);
            }
            if (!share.more(count)) break;
            const uint32_t i = share.take(count, (uint32_t)__popc(m_idle),
                                          (uint32_t)__popc(m_idle & ((1u << lane) - 1u)), fetch);
            if (idle && i < count) {
                idx = i;
                const float4 q0 = qload<NC>(&q[stride * (size_t)idx]);
                const float4 q1 = qload<NC>(&q[stride * (size_t)idx + 1]);
                trav_init<ANY>(S, s, xyz(q0), xyz(q1), ANY ? q0.w : 0.0f);
                st.clear();
                have = true;
            }
            steps = 0;
            continue;
        }
        if (++steps > guard) {  // a malformed tree: report and stop
            overflow = true;
            s.cur = TRAV_IDLE;
            continue;
        }
#pragma unroll
        for (int u = 0; u < TRACE_NODE_STEPS; ++u) {
            if (s.cur >= 0 && s.cur != TRAV_IDLE) {
                if ((uint32_t)s.cur >= S.n_nodes) {  // corrupt reference
                    overflow = true;
                    s.cur = TRAV_IDLE;
                } else {
                    if (COUNT) tc.nodes++;
                    int32_t first;
                    if (visit4<ANY>(S.nodes + BVH_NODE_F4 * (size_t)s.cur, s.r, s.t_best, first, st, overflow))
                        s.cur = first;
                    else
                        trav_pop<ANY>(s, st);
                }
            }
        }
        if (s.cur < 0) {
            if (trav_leaf<ANY, COUNT>(S, s, ~(uint32_t)s.cur, tc)) {
                s.hit = true;
                s.cur = TRAV_IDLE;
            } else {
                trav_pop<ANY>(s, st);
            }
        }
    }
    if (overflow) atomicAdd(err_stack, 1u);
    if (COUNT) {
        // one addition per warp that has something to add: every warp of the grid
        // comes by here, whatever the queue's length, and the additions to one
        // counter complete one after the other (2 ms a frame of any size by lane)
        unsigned long long nodes = tc.nodes, tris = tc.tris;
        for (int o = 16; o > 0; o >>= 1) {
            nodes += __shfl_down_sync(full, nodes, o);
            tris += __shfl_down_sync(full, tris, o);
        }
        if (lane == 0 && nodes) atomicAdd((unsigned long long*)&stats[0], nodes);
        if (lane == 0 && tris) atomicAdd((unsigned long long*)&stats[1], tris);
    }
}

// Queue slot of a frame -> pixel.  Slots go by 32 over 8x4 pixel tiles
// (tiles row by row), so the camera rays a traversal warp fetches together
// cover a compact patch of the screen and walk nearly the same nodes; the
// right and bottom strips the tiles leave (width % 8, height % 4) follow
// row by row.  A bijection on [0, w * h).
__device__ __forceinline__ uint32_t slot_pixel(uint32_t s, uint32_t w, uint32_t h) {
    const uint32_t tx = w >> 3, h4 = h & ~3u;
    const uint32_t tiled = tx * 8u * h4;
    if (s < tiled) {
        const uint32_t t = s >> 5, l = s & 31u;
        const uint32_t ty = t / tx, tt = t - ty * tx;
        return (ty * 4u + (l >> 3)) * w + tt * 8u + (l & 7u);
    }
    s -= tiled;
    const uint32_t rw = w - tx * 8u;
    if (s < rw * h4) {
        const uint32_t y = s / rw;
        return y * w + tx * 8u + (s - y * rw);
    }
    return h4 * w + (s - rw * h4);
}

// Queue slot of a wavefront of `frames` frames -> (frame, pixel): tile by tile,
// each tile's 32 pixels in every frame before the next tile's, so the rays in
// flight at a time start from a small part of the screen and share the tree's
// nodes in the caches; the strips the tiles leave follow frame by frame.
__device__ __forceinline__ void slot_path(uint32_t s, uint32_t w, uint32_t h, uint32_t frames, uint32_t& fr,
                                          uint32_t& pixel) {
    const uint32_t tiled = (w >> 3) * 8u * (h & ~3u), pixels = w * h;
    if (s < tiled * frames) {
        const uint32_t t = s / (32u * frames), r = s - t * 32u * frames;
        fr = r >> 5;
        pixel = slot_pixel(32u * t + (r & 31u), w, h);
    } else {
        const uint32_t strip = pixels - tiled;
        s -= tiled * frames;
        fr = s / strip;
        pixel = slot_pixel(tiled + (s - fr * strip), w, h);
    }
}

// Closest hits of one warp's 32 rays walked as a packet (packet_visit4):
// every lane of the warp calls it together; a lane with valid = false takes
// part in the walk but accepts no box.  On return s holds the lane's hit as
// trav_init and trav_leaf leave it (t_best, best_prim, best_key).
__device__ __forceinline__ void packet_closest(const DeviceScene& S, f3 o, f3 d, bool valid, TravState& s,
                                               int32_t* st_ref, float* st_t, bool& overflow) {
    trav_init<false>(S, s, o, d, 0.0f);
    // a lane past the end of the queue, or whose ray walks no tree, accepts no
    // box (t_f <= -1 < t_n)
    const bool walks = valid && s.cur == 0;
    const float t_planes = s.t_best;
    if (!walks) s.t_best = -1.0f;
    int sp = 0;
    int32_t cur = 0;
    uint32_t guard = 2u * S.n_nodes + 64u;
    bool live = S.n_nodes != 0;
    while (live) {
        if (cur >= 0) {
            if (--guard == 0u || (uint32_t)cur >= S.n_nodes) { overflow = true; break; }
            int32_t first;
            if (packet_visit4(S.nodes + BVH_NODE_F4 * (size_t)cur, s.r, s.t_best, first, st_ref, st_t, sp,
                              overflow))
                cur = first;
            else live = packet_pop(s.t_best, st_ref, st_t, sp, cur);
        } else {
            TraceCounters tc;
            if (walks) trav_leaf<false, false>(S, s, ~(uint32_t)cur, tc);
            live = packet_pop(s.t_best, st_ref, st_t, sp, cur);
        }
    }
    if (!walks) s.t_best = t_planes;
}

// Closest hits of a coherent queue as warp packets (packet_visit4): each
// warp takes 32 consecutive entries, which the camera kernel fills from
// one 8x4 pixel tile, and walks the tree once for all of them.  The
// entries, their hits and done(i, state) are those of persistent_trace;
// only the traversal order differs, which the closest hit does not depend
// on.  No traversal counters (instrumented frames use persistent_trace).
template <bool NC = true, typename Done>
__device__ __forceinline__ void packet_trace(const DeviceScene& S, const float4* __restrict__ q, uint32_t stride,
                                             uint32_t count, uint32_t* fetch, uint32_t* err_stack, Done done) {
    const unsigned full = 0xffffffffu;
    const uint32_t lane = lane_id();
    int32_t st_ref[CUPBR_STACK_SIZE];
    float st_t[CUPBR_STACK_SIZE];
    bool overflow = false;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(fetch, 32u);
        base = __shfl_sync(full, base, 0);
        if (base >= count) break;
        const uint32_t idx = base + lane;
        const bool valid = idx < count;
        f3 o = mk(0.0f, 0.0f, 0.0f), d = mk(0.0f, 0.0f, 1.0f);
        if (valid) {
            o = xyz(qload<NC>(&q[stride * (size_t)idx]));
            d = xyz(qload<NC>(&q[stride * (size_t)idx + 1]));
        }
        TravState s;
        packet_closest(S, o, d, valid, s, st_ref, st_t, overflow);
        if (valid) done(idx, s);
    }
    if (overflow) atomicAdd(err_stack, 1u);
}

}  // namespace cupbr_b200
