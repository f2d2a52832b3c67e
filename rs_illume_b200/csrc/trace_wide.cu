// Wide-BVH ray queries (W = 4 or 8 children per node); the traversal state
// is WideTracer (wide_tracer.cuh).
//
// Schedules:
//  * grid: one thread per ray.
//  * persistent (default): a grid sized to fill the GPU once; each warp claims
//    rays 64 at a time (32 for short queues) from a device counter and hands
//    them to lanes that are free.  A claimed ray is first tested against the
//    scene's root box; rays that miss it (most incoherent rays) are answered
//    at once and never occupy a lane (see k_trace_wide_persistent's kPool for
//    the two ways of doing so).  Each loop iteration advances every busy lane
//    by exactly one node or one leaf, then refills finished lanes, so a warp
//    stays full while its rays differ in length.
//  * split tail (pooled persistent kernel once every ray is claimed, and the
//    one-thread-per-ray kernel k_trace_wide_split throughout): idle lanes
//    take stacked subtrees of their warp's unfinished rays (share_subtrees in
//    wide_tracer.cuh), so a launch does not wait on its longest rays alone.
#include <algorithm>

#include "wide_tracer.cuh"

namespace ilm {

namespace {

template <int W, int kStack, bool kAny, bool kAnalytic>
__global__ void __launch_bounds__(128) k_trace_wide(TraceArgs a) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ray_count(a)) return;
    RayIn r = load_ray(a.rays, i);
    using Tracer = WideTracer<W, kStack, kAny, kAnalytic>;
    typename Tracer::Entry stk[Tracer::kDepth];
    Tracer T(stk);
    T.init(r);
    if (a.n_nodes == 0 || !T.enters(a.bound)) { write_miss(i, r, a.hits, a.occ); return; }
    while (!T.step(a)) {}
    T.write(i, a);
}

// Rays a warp starts with where each ray has a lane of its own, for n rays on a
// launch of `threads` resident threads.  The other lanes start idle and take
// subtrees of the warp's rays, so fewer rays a warp shorten the longest ray's
// chain of steps; but more warps share the SMs' issue slots, and helpers
// traverse some of what the lone ray would have culled, which weighs more the
// more rays there are.
// A path queue takes the smallest power of two (at most 32) whose warps are all
// resident at once: its rays are coherent, and nearly all enter the scene.
__host__ __device__ __forceinline__ uint32_t queue_rays_per_warp(uint64_t n, uint64_t threads) {
    uint32_t r = 1;
    while (r < 32u && n * 32u > threads * r) r *= 2u;
    return r;
}
// A query takes r rays a warp while they need at most (16 - r) / 16 of the
// wave's warps: 1 up to 3,885 rays on 148 SMs of 7 blocks, 2 up to 7,252, 4 up
// to 12,432, 8 up to 16,576, then 16, and 32 where 16 would not all be resident
// (66,304).  Against 16 a warp (closest hit, six scenes, camera and incoherent
// rays): 32 rays 1.36 times as fast, 1,000 1.42, 8,000 1.24, 16,000 1.09.
// Where 8 a warp would still fit, 20,000 to 33,000 rays, camera rays gain 1.1
// by it but incoherent ones lose up to 15 %.  us at 32 / 16 / chosen, camera
// rays on a 32,768-triangle soup: 1,000 rays 84 / 59 / 31, 8,000 101 / 66 / 40,
// 16,000 107 / 70 / 54.
inline uint32_t rays_per_warp(uint64_t n, uint64_t threads) {
    const uint64_t warps = threads / 32u;
    if (n > 16u * warps) return 32u;
    uint32_t r = 1;
    while (r < 16u && 16u * n > warps * r * (16u - r)) r *= 2u;
    return r;
}

// One thread per ray with the split tail from the start: a lane whose ray
// missed the scene's root box or has finished takes subtrees of its warp's
// unfinished rays (share_subtrees).  A one-wave query is all tail: its
// launch lasts as long as its longest rays.
// Lane `lane` < warp_rays of warp w starts on ray w * warp_rays + lane; the
// other lanes start idle and help from the first pass.
template <int W, int kStack, bool kAny, bool kAnalytic>
__device__ __forceinline__ void trace_split(const TraceArgs& a, const uint64_t n, const uint32_t warp_rays,
                                            uint32_t* warp_words) {
    const unsigned lane = threadIdx.x & 31u;
    uint32_t* ids = warp_words + kPoolWords;
    using Tracer = WideTracer<W, kStack, kAny, kAnalytic>;
    typename Tracer::Entry stk[Tracer::kDepth];
    Tracer T(stk);
    uint32_t st = kFree | (lane << 2);
    const uint64_t warp_id = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t i = warp_id * warp_rays + lane;
    if (lane < warp_rays && i < n) {
        const RayIn r = load_ray(a.rays, i);
        T.init(r);
        if (a.n_nodes != 0 && T.enters(a.bound)) {
            ids[2 * lane] = (uint32_t)i;
            ids[2 * lane + 1] = (uint32_t)(i >> 32);
            st = kOwner | (lane << 2);
        } else {
            write_miss(i, r, a.hits, a.occ);
        }
    }
    for (;;) {
        bool owner_occluded = kAny && __shfl_sync(0xFFFFFFFFu, (int)T.occluded, owner_of(st));
        share_subtrees<Tracer, kAny>(T, st, owner_occluded, warp_words);
        if (kAny) owner_occluded = __shfl_sync(0xFFFFFFFFu, (int)T.occluded, owner_of(st));
        if (!__any_sync(0xFFFFFFFFu, role_of(st) != kFree)) break;
        const uint32_t role = role_of(st);
        bool done = false;
        if ((role == kOwner || role == kHelper) && owner_occluded) done = true;
        else if (role == kOwner || role == kHelper) done = T.step(a);
        const unsigned fin = __ballot_sync(0xFFFFFFFFu, role == kHelper && done);
        if (fin) merge_helpers<Tracer, kAny>(T, st, fin);
        if (role == kHelper && done) st = kFree | (lane << 2);
        if (role == kOwner && done) st = (st & ~3u) | kWaiting;
        if (role_of(st) == kWaiting && (st >> 8) == 0u) {
            T.write((uint64_t)ids[2 * lane] | ((uint64_t)ids[2 * lane + 1] << 32), a);
            st = kFree | (lane << 2);
        }
    }
}

template <int W, int kStack, bool kAny, bool kAnalytic>
__global__ void __launch_bounds__(128) k_trace_wide_split(TraceArgs a) {
    __shared__ __align__(16) uint32_t s_warp[4][kWarpWords];
    trace_split<W, kStack, kAny, kAnalytic>(a, ray_count(a), a.warp_rays, s_warp[threadIdx.x >> 5]);
}

// Persistent schedule, pooled refill: the whole warp tests each claimed chunk
// against the root box, two rays per lane, answers the misses at full width,
// and keeps the rays that enter in a per-warp pool in shared memory; idle
// lanes take rays from the pool.  For incoherent batches most rays miss the
// scene, and this keeps the lanes that are still traversing from waiting
// while a few idle lanes test misses one at a time (5,330 against 4,420
// Mrays/s on the 2M-ray ball workload).  It carries the split tail.
template <int W, int kStack, bool kAny, bool kAnalytic, bool kShortClaims>
__device__ __forceinline__ void trace_pooled(const TraceArgs& a, const uint64_t n, uint32_t* warp_words) {
    // A short queue (fewer than two rays per resident lane) is claimed one ray
    // per lane, so that its rays run side by side rather than two per lane.
    const unsigned chunk = kShortClaims || n < 2ull * gridDim.x * blockDim.x ? 32u : kChunk;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    using Tracer = WideTracer<W, kStack, kAny, kAnalytic>;
    typename Tracer::Entry stk[Tracer::kDepth];
    Tracer T(stk);
    bool exhausted = false;                             // warp-uniform
    uint32_t* pool = warp_words;                    // offsets of the pooled rays in their chunk
    uint32_t* ids = warp_words + kPoolWords;        // each lane's ray id (owners)
    unsigned pool_n = 0;                            // warp-uniform
    unsigned long long pool_base = 0;               // warp-uniform: the pooled rays' chunk
    uint32_t st = kFree | (lane << 2);
    for (;;) {
        if (!exhausted) {
            unsigned need = __ballot_sync(0xFFFFFFFFu, role_of(st) == kFree);
            // Every pass either hands out pooled rays or claims and filters
            // a chunk (claims are only made with an empty pool), so the
            // loop ends.
            while (need != 0u) {
                if (pool_n == 0) {
                    unsigned long long b = 0;
                    if (lane == 0) b = atomicAdd(a.counter, (unsigned long long)chunk);
                    b = __shfl_sync(0xFFFFFFFFu, b, 0);
                    if (b >= n) { exhausted = true; break; }
                    for (unsigned k = 0; k < chunk; k += 32u) {
                        const uint64_t rid = b + k + lane;
                        bool enter = false;
                        if (rid < n) {
                            const RayIn r = load_ray(a.rays, rid);
                            enter = a.n_nodes != 0 && root_enters(r, a.bound);
                            if (!enter) write_miss(rid, r, a.hits, a.occ);
                        }
                        const unsigned m = __ballot_sync(0xFFFFFFFFu, enter);
                        if (enter) pool[pool_n + __popc(m & below)] = k + lane;
                        pool_n += __popc(m);
                    }
                    __syncwarp();
                    pool_base = b;
                    continue;
                }
                const unsigned rank = __popc(need & below);
                const unsigned take = min((unsigned)__popc(need), pool_n);
                if (((need >> lane) & 1u) && rank < take) {
                    const uint64_t id = pool_base + pool[pool_n - 1u - rank];
                    ids[2 * lane] = (uint32_t)id;
                    ids[2 * lane + 1] = (uint32_t)(id >> 32);
                    T.init(load_ray(a.rays, id));
                    st = kOwner | (lane << 2);
                }
                pool_n -= take;
                __syncwarp();
                need = __ballot_sync(0xFFFFFFFFu, role_of(st) == kFree);
            }
        }
        // Subtrees are shared once the counter has run out (warp-uniform).
        // Before that every busy lane is an owner, and the closest-hit
        // kernel skips the helpers' bookkeeping (measured 1 % faster); the
        // any-hit kernel keeps it throughout (2 % faster that way).
        const bool split_now = exhausted && a.split_tail;
        const bool tail = kAny || split_now;
        // A helper of an occluded any-hit ray has nothing left to find.
        bool owner_occluded = kAny && __shfl_sync(0xFFFFFFFFu, (int)T.occluded, owner_of(st));
        if (split_now) {
            share_subtrees<Tracer, kAny>(T, st, owner_occluded, warp_words);
            // Lanes that just took a subtree have a new owner.
            if (kAny) owner_occluded = __shfl_sync(0xFFFFFFFFu, (int)T.occluded, owner_of(st));
        }
        if (!__any_sync(0xFFFFFFFFu, role_of(st) != kFree)) break;   // only once exhausted
        const uint32_t role = role_of(st);
        bool done = false;
        // An any-hit ray one of its helpers found occluded is finished.
        if ((role == kOwner || role == kHelper) && owner_occluded) done = true;
        else if (role == kOwner || role == kHelper) done = T.step(a);
        if (tail) {
            const unsigned fin = __ballot_sync(0xFFFFFFFFu, role == kHelper && done);
            if (fin) merge_helpers<Tracer, kAny>(T, st, fin);
            if (role == kHelper && done) st = kFree | (lane << 2);
            if (role == kOwner && done) st = (st & ~3u) | kWaiting;
            if (role_of(st) == kWaiting && (st >> 8) == 0u) {
                T.write((uint64_t)ids[2 * lane] | ((uint64_t)ids[2 * lane + 1] << 32), a);
                st = kFree | (lane << 2);
            }
        } else if (done) {
            T.write((uint64_t)ids[2 * lane] | ((uint64_t)ids[2 * lane + 1] << 32), a);
            st = kFree | (lane << 2);
        }
    }
}

// Persistent schedule, lane refill: each idle lane tests its own claims,
// repeating until one enters (ILM_FLAG_LANE_REFILL); no split tail.
template <int W, int kStack, bool kAny, bool kAnalytic>
__device__ __forceinline__ void trace_lanes(const TraceArgs& a, const uint64_t n) {
    // A short queue (fewer than two rays per resident lane) is claimed one ray
    // per lane, so that its rays run side by side rather than two per lane.
    const unsigned chunk = n < 2ull * gridDim.x * blockDim.x ? 32u : kChunk;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    using Tracer = WideTracer<W, kStack, kAny, kAnalytic>;
    typename Tracer::Entry stk[Tracer::kDepth];
    Tracer T(stk);
    bool exhausted = false;                             // warp-uniform
    bool active = false;
    uint64_t id = 0;
    unsigned long long chunk_next = 0, chunk_end = 0;   // warp-uniform
    for (;;) {
        unsigned need = __ballot_sync(0xFFFFFFFFu, !active);
        // Hand rays to idle lanes; rays missing the root box are answered here.
        // Every pass hands out >= 1 ray or claims a chunk, so the loop ends.
        while (need != 0u && !exhausted) {
            if (chunk_next == chunk_end) {
                unsigned long long b = 0;
                if (lane == 0) b = atomicAdd(a.counter, (unsigned long long)chunk);
                b = __shfl_sync(0xFFFFFFFFu, b, 0);
                if (b >= n) { exhausted = true; break; }
                chunk_next = b;
                chunk_end = b + chunk < n ? b + chunk : n;
            }
            unsigned avail = (unsigned)(chunk_end - chunk_next);
            unsigned rank = __popc(need & below);
            if (((need >> lane) & 1u) && rank < avail) {
                id = chunk_next + rank;
                RayIn r = load_ray(a.rays, id);
                T.init(r);
                if (a.n_nodes != 0 && T.enters(a.bound)) active = true;
                else write_miss(id, r, a.hits, a.occ);
            }
            chunk_next += min((unsigned)__popc(need), avail);
            need = __ballot_sync(0xFFFFFFFFu, !active);
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;   // only reached once exhausted
        if (active && T.step(a)) {
            T.write(id, a);
            active = false;
        }
    }
}

// kMinBlocks asks the compiler for that many resident 128-thread blocks
// per SM (launch_refill).
template <int W, int kStack, bool kAny, int kMinBlocks, bool kAnalytic, bool kPool>
__global__ void __launch_bounds__(128, kMinBlocks) k_trace_wide_persistent(TraceArgs a) {
    if constexpr (kPool) {
        __shared__ __align__(16) uint32_t s_warp[4][kWarpWords];
        const uint64_t n = ray_count(a);
        // An empty queue.  (Without this return the loop compiles to something
        // else: 2,000,003 shadow rays on 1.3M triangles 190.1 us, 188.1 with it.)
        if (n == 0) return;
        trace_pooled<W, kStack, kAny, kAnalytic, W == 8 && kMinBlocks == 1 && !kAnalytic>(
            a, n, s_warp[threadIdx.x >> 5]);
    } else {
        trace_lanes<W, kStack, kAny, kAnalytic>(a, ray_count(a));
    }
}

// A path queue, whose count is known on the device only: at most one ray per
// thread of the launch runs with the split tail from the start (all of its
// rays resident at once), a larger count on the pooled schedule.  As two
// launches, one of which returned at once, and a memset of the work counter
// before each persistent one, a bounce was nine launches of which five did
// next to nothing.
template <int W, int kStack, bool kAny>
__global__ void __launch_bounds__(128, 7) k_trace_wide_queue(TraceArgs a) {
    __shared__ __align__(16) uint32_t s_warp[4][kWarpWords];
    uint32_t* warp_words = s_warp[threadIdx.x >> 5];
    const uint64_t n = ray_count(a), threads = (uint64_t)gridDim.x * blockDim.x;
    if (n <= threads) trace_split<W, kStack, kAny, false>(a, n, queue_rays_per_warp(n, threads), warp_words);
    else trace_pooled<W, kStack, kAny, false, false>(a, n, warp_words);
}

template <int W, int kStack, int kMinBlocks, bool kAnalytic, bool kPool>
cudaError_t launch_persistent(const TraceArgs& t, cudaStream_t s) {
    const unsigned block = 128;
    auto kc = k_trace_wide_persistent<W, kStack, false, kMinBlocks, kAnalytic, kPool>;
    auto ka = k_trace_wide_persistent<W, kStack, true, kMinBlocks, kAnalytic, kPool>;
    uint64_t grid = resident_blocks(t.occ ? (const void*)ka : (const void*)kc, (int)block);
    if (grid == 0) return cudaErrorInvalidConfiguration;
    const uint64_t need_blocks = (t.n + block - 1) / block;
    if (grid > need_blocks) grid = need_blocks;
    if (!t.counter_ready) {
        cudaError_t e = cudaMemsetAsync(t.counter, 0, sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
    }
    if (t.occ) ka<<<(unsigned)grid, block, 0, s>>>(t);
    else kc<<<(unsigned)grid, block, 0, s>>>(t);
    return cudaGetLastError();
}

// Persistent launch of either refill: by the build for many resident blocks
// per SM (the pooled kernel at 7, whose split tail's state fits 72 registers;
// the lane-refill kernel at 8, 64 registers) or with
// the compiler's registers (triangles alone 112 to 122 at width 8, four blocks,
// and 72 to 90 at width 4; with analytic shapes 112 to 128, where the other
// build spills up to 242 bytes).  The caller's flag asks for the first; without
// it, a query on triangles alone takes it from six rays per thread of its wave
// on (795,648 rays on 148 SMs), lane refill from three.  Long queries have
// latency to hide all the time: 2,000,000 rays on triangles 1.14 times as fast
// (closest hit and any hit, six scenes, camera and incoherent rays), 1,000,000
// 1.06.  In short ones more of the launch is its longest rays, and those run
// faster with fewer warps beside them: 500,000 incoherent rays on 327,680
// triangles 104 us against 117, 130,000 64 against 71, and at 700,000 one query
// in three is still slower.  There the width-8 kernel with the compiler's
// registers claims 32 rays at a time, one a lane: with 64, 200,000 camera rays
// took 152 us (140 now), since its 2,368 warps claim 1.3 times each.
constexpr int kPooledBlocks = 7, kLaneBlocks = 8;
template <int W, int kStack>
uint64_t deep_query(bool pooled) {
    const uint64_t threads =
        128u * resident_blocks((const void*)k_trace_wide_persistent<W, kStack, false, kPooledBlocks, false, true>, 128);
    return (pooled ? 6u : 3u) * threads;
}

template <int W, int kStack, bool kAnalytic>
cudaError_t launch_refill(const TraceArgs& t, const LaunchParams& lp, cudaStream_t s) {
    if (lp.high_occupancy || (!kAnalytic && t.n >= deep_query<W, kStack>(lp.root_pool != 0)))
        return lp.root_pool ? launch_persistent<W, kStack, kPooledBlocks, kAnalytic, true>(t, s)
                            : launch_persistent<W, kStack, kLaneBlocks, kAnalytic, false>(t, s);
    return lp.root_pool ? launch_persistent<W, kStack, 1, kAnalytic, true>(t, s)
                        : launch_persistent<W, kStack, 1, kAnalytic, false>(t, s);
}

template <int W, int kStack, bool kAnalytic>
cudaError_t launch_variant(const TraceArgs& t, const LaunchParams& lp, cudaStream_t s) {
    const unsigned block = 128;
    if (lp.persistent && t.counter) {
        if constexpr (!kAnalytic) {
            if (lp.queue_split && t.n_dev && t.split_tail) {
                auto kc = k_trace_wide_queue<W, kStack, false>;
                auto ka = k_trace_wide_queue<W, kStack, true>;
                // a warp for every ray that the queue can hold, up to one wave
                const uint64_t grid =
                    std::min<uint64_t>(resident_blocks(t.occ ? (const void*)ka : (const void*)kc, (int)block),
                                       (t.n + block / 32 - 1) / (block / 32));
                if (grid == 0) return cudaErrorInvalidConfiguration;
                if (!t.counter_ready) {
                    cudaError_t e = cudaMemsetAsync(t.counter, 0, sizeof(unsigned long long), s);
                    if (e != cudaSuccess) return e;
                }
                if (t.occ) ka<<<(unsigned)grid, block, 0, s>>>(t);
                else kc<<<(unsigned)grid, block, 0, s>>>(t);
                return cudaGetLastError();
            }
        }
        return launch_refill<W, kStack, kAnalytic>(t, lp, s);
    }
    unsigned grid = (unsigned)((t.n + block - 1) / block);
    if (t.split_tail) {
        auto kc = k_trace_wide_split<W, kStack, false, kAnalytic>;
        auto ka = k_trace_wide_split<W, kStack, true, kAnalytic>;
        const uint64_t wave = resident_blocks(t.occ ? (const void*)ka : (const void*)kc, (int)block) * block;
        TraceArgs q = t;
        q.warp_rays = rays_per_warp(t.n, wave);
        const uint64_t rays_per_block = (uint64_t)q.warp_rays * (block / 32);
        const unsigned g = (unsigned)((t.n + rays_per_block - 1) / rays_per_block);
        if (t.occ) ka<<<g, block, 0, s>>>(q);
        else kc<<<g, block, 0, s>>>(q);
        return cudaGetLastError();
    }
    if (t.occ) k_trace_wide<W, kStack, true, kAnalytic><<<grid, block, 0, s>>>(t);
    else k_trace_wide<W, kStack, false, kAnalytic><<<grid, block, 0, s>>>(t);
    return cudaGetLastError();
}

// Accels without quadric or curve records run the triangle-only variants.
template <int W, int kStack>
cudaError_t launch(const TraceArgs& t, const LaunchParams& lp, cudaStream_t s) {
    return t.spheres ? launch_variant<W, kStack, true>(t, lp, s) : launch_variant<W, kStack, false>(t, lp, s);
}

}  // namespace

uint64_t wide_grid_wave(int width, int stack_depth) {
    const bool w8 = width == 8, deep = stack_depth > 32;
    const void* k = w8 ? (deep ? (const void*)k_trace_wide<8, 64, false, true> : (const void*)k_trace_wide<8, 32, false, true>)
                       : (deep ? (const void*)k_trace_wide<4, 64, false, true> : (const void*)k_trace_wide<4, 32, false, true>);
    return resident_blocks(k, 128) * 128u;
}

uint64_t wide_deep_query(int width, const LaunchParams& lp) {
    const bool deep = lp.stack_depth > 32, pooled = lp.root_pool != 0;
    return width == 8 ? (deep ? deep_query<8, 64>(pooled) : deep_query<8, 32>(pooled))
                      : (deep ? deep_query<4, 64>(pooled) : deep_query<4, 32>(pooled));
}

cudaError_t launch_trace_wide(int width, const TraceArgs& t, const LaunchParams& lp, cudaStream_t s) {
    bool deep = lp.stack_depth > 32;
    if (width == 8) return deep ? launch<8, 64>(t, lp, s) : launch<8, 32>(t, lp, s);
    return deep ? launch<4, 64>(t, lp, s) : launch<4, 32>(t, lp, s);
}

}  // namespace ilm
