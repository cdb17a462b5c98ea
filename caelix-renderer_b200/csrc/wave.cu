// The wavefront trace (trace.cuh): path state in HBM, one kernel per stage over compacted queues.
//
// Stages of one sub-wave (a range of the pixels of one sample index, or every pixel of several):
//   wave_generate_kernel  one slot per pixel and sample: the camera ray (trace_pixel's), queued;
//   then bounce_count + 1 times:
//   wave_trace_kernel     every queued ray: the closest hit (extension rays) or occlusion (shadow
//                         rays) through the brick-grid DDA, written to the slot
//                         (wave_trace_refill_kernel in large waves, after the camera rays);
//   wave_shade_kernel     every live path: its shadow result, then its vertex (the per-frame
//                         kernel's integrator step without the light tree: emission, albedo,
//                         Russian roulette), queueing its extension ray, its light draw and its
//                         lamp weight; a finished path adds its sample to the pixel (the last
//                         sample divides), or leaves it in its slot where several samples of a
//                         pixel are in flight;
//   wave_light_kernel     every queued light draw (light-tree NEE, queueing its shadow ray) and
//                         every queued lamp hit (its MIS weight, then its emission);
//   and with several samples wave_resolve_kernel: their sums in sample order.
// A path's arithmetic is trace_pixel's in the same order (the shadow contribution of a vertex is
// added before anything of the next vertex), so the radiance is the per-frame kernel's, bit for
// bit. Queues are compacted with warp-aggregated atomics; every kernel reads its queue length on
// the device, so a whole frame is recorded without a host synchronisation (graph-capturable).
//
// Figures beside a part are its own before and after, in the state of the file when it was made (one B200). The
// frames they name now take: 160 x 90 0.108 ms, 512 x 512 0.405, 333 x 251 x 8 spp 0.709, 1920 x 1080 x 4 spp on
// 300 k bricks 9.4, the adjoint of 256 x 256 x 8 spp 1.81, 12 views of 256 and 512 squared 4.73.
#include <algorithm>
#include <mutex>
#include <cstdint>
#include <type_traits>

#include "launch.cuh"
#include "trace.cuh"
#include "trace_device.cuh"

namespace cx {

namespace {

constexpr uint32_t kWaveThreads = 128;
constexpr uint32_t kKindPrimary = 0, kKindBounce = 1, kKindShadow = 2;
constexpr uint32_t kSlotMask = 0x3FFFFFFFu;
constexpr uint32_t kFlagBounce = 0xFFu;       // bounce_index
constexpr uint32_t kFlagSegLight = 1u << 8;   // segment_light = 3
constexpr uint32_t kFlagShadow = 1u << 9;     // a shadow ray of the last vertex was queued
constexpr uint32_t kFlagExt = 1u << 10;       // an extension ray was queued
constexpr uint32_t kFlagPrimary = 1u << 11;   // that extension ray is the camera ray
constexpr uint32_t kLampEnds = 1u << 31;      // of a lampq entry: the path ends with this emission
// The counters in WaveBuffers::counts: 0..3 the queue lengths of the two parities (rays, paths), then
// the trace and shade launches' fetch counters of the two parities, the lengths of the light draw
// and lamp queues and the light launch's fetch counter (cleared by the next trace launch). Each has a
// 128-byte line of its own: an atomic takes about a nanosecond at its address, and a launch over 8 M
// paths made a million of them side by side. With lines of their own, appends of 128 entries at a time,
// chunks of up to 256 items and rays counted per warp (one B200, 1920 x 1080 x 4 spp on 300 k bricks): the
// first shade launch 731 -> 236 us, all of them 2.25 -> 0.94 ms, the camera rays' generation 394 -> 71 us, the
// frame 12.1 -> 11.1 ms; 512 x 512 0.456 -> 0.424, 160 x 90 0.125 -> 0.117, 12 batched views 5.23 -> 4.72.
constexpr uint32_t kFetchTrace = 4, kFetchShade = 6, kCountNee = 8, kCountLamp = 9, kFetchLight = 10;
constexpr uint32_t kCounters = 11;
constexpr uint32_t kCounterStride = 32;
constexpr uint32_t kCountWords = kCounters * kCounterStride;
__device__ __forceinline__ uint32_t* counter_of(const WaveBuffers& b, uint32_t k) { return b.counts + k * kCounterStride; }
__device__ __forceinline__ uint32_t count_of(const WaveBuffers& b, uint32_t k)
{
    return *(volatile uint32_t*)counter_of(b, k);
}

// The items of a queue of n that the calling warp works on, taken `chunk` at a time from a fetch counter:
// the work of a launch whose items' costs differ widely spreads over the warps until its end. Every lane
// calls.
struct WarpRange
{
    uint32_t at, end;
    // Whether items [at, end) remain (a new chunk where the last one is done).
    __device__ __forceinline__ bool more(uint32_t* counter, uint32_t n, uint32_t chunk)
    {
        if (at < end) return true;
        uint32_t base = 0;
        if ((threadIdx.x & 31u) == 0) base = atomicAdd(counter, chunk);
        at = __shfl_sync(0xFFFFFFFFu, base, 0);
        end = min(at + chunk, n);
        return at < end;
    }
};
// The chunk: an eighth of a warp's share of the items, in whole warps, 32 to 256.
__device__ __forceinline__ uint32_t chunk_for(uint32_t n)
{
    const uint32_t share = n / (8u * gridDim.x * (blockDim.x / 32u));
    return min(max(share & ~31u, 32u), 256u);
}

struct WaveGen
{
    const uint32_t* table;  // entries (view | sample << 16, of the wave), then item bases (`entries` each)
    uint32_t entries;
    uint32_t first_sample;  // the entries' samples count from it
    uint32_t samples;       // sample indices of the wave
    uint32_t first_item;
    uint32_t count;
    uint32_t block_width;
};

// A warp's appends to a queue, collected in shared memory and written 128 at a time (one atomic, whole
// lines). Every lane calls; finish() writes the rest.
constexpr uint32_t kQueueBatch = 128;
struct WarpQueue
{
    uint32_t* buffer;  // kQueueBatch + 32 words of this warp
    uint32_t* counter;
    uint32_t* queue;
    uint32_t held = 0;
    __device__ __forceinline__ void write(uint32_t n)
    {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(counter, n);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        __syncwarp();
        for (uint32_t j = lane; j < n; j += 32) queue[base + j] = buffer[j];
    }
    __device__ __forceinline__ void push(bool has, uint32_t value)
    {
        const uint32_t who = __ballot_sync(0xFFFFFFFFu, has);
        if (has) buffer[held + (uint32_t)__popc(who & lanemask_lt())] = value;
        held += (uint32_t)__popc(who);
        if (held < kQueueBatch) return;
        write(kQueueBatch);
        held -= kQueueBatch;
        const uint32_t rest = buffer[kQueueBatch + (threadIdx.x & 31u)];
        __syncwarp();
        if ((threadIdx.x & 31u) < held) buffer[threadIdx.x & 31u] = rest;
        __syncwarp();
    }
    __device__ __forceinline__ void finish()
    {
        if (held) write(held);
        held = 0;
    }
};
constexpr uint32_t kQueueWords = kQueueBatch + 32;

// The entry (of the first `entries` of a wave) that holds item `item`, and the item within it.
__device__ __forceinline__ uint32_t wave_entry(const WaveGen& g, uint32_t entries, uint32_t item, uint32_t& local)
{
    const uint32_t* bases = g.table + g.entries;
    uint32_t lo = 0, hi = entries;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(bases + mid) <= item) lo = mid;
        else hi = mid;
    }
    local = item - __ldg(bases + lo);
    return lo;
}

__global__ void __launch_bounds__(kWaveThreads)
    wave_generate_kernel(const WaveView* __restrict__ views, const WaveGen g, const WaveBuffers b)
{
    const uint32_t i = blockIdx.x * kWaveThreads + threadIdx.x;
    const uint32_t bw = g.block_width, bh = 32u / bw;
    // Every item has its place in the first queues, those outside the image a hole: no counting (two
    // atomics per warp on the queue lengths took four fifths of this kernel over 8 M paths).
    if (i == 0) *counter_of(b, 0) = *counter_of(b, 1) = g.count;
    if (i < g.count) {
        bool valid = false;
        const uint32_t item = g.first_item + i;
        uint32_t local;
        const uint32_t vs = __ldg(g.table + wave_entry(g, g.entries, item, local));
        const WaveView& V = views[vs & 0xFFFFu];
        const TraceParams& P = V.params;
        const uint32_t blk = local >> 5, in = local & 31u;
        const uint32_t px = (blk % V.blocks_x) * bw + in % bw;
        const uint32_t py = (blk / V.blocks_x) * bh + in / bw;
        if (px < P.width && py < P.height) {
            valid = true;
            const float sx = (float)px + 0.5f + 0.0f;
            const float sy = (float)py + 0.5f + 0.0f;
            const float ndc_x = sx / (float)P.width * 2.0f - 1.0f;
            const float ndc_y = 1.0f - sy / (float)P.height * 2.0f;
            const float a = ndc_x * P.tan_half_fov_y * P.aspect;
            const float bb = ndc_y * P.tan_half_fov_y;
            float d[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) d[k] = P.right[k] * a + P.up[k] * bb + P.forward[k];
            const float inv_len = 1.0f / sqrtf(dot3(d, d));
#pragma unroll
            for (int k = 0; k < 3; ++k) d[k] = d[k] * inv_len;
            b.item[i] = py * P.width + px;
            b.vs[i] = vs;
            b.flags[i] = kFlagExt | kFlagPrimary;
            b.org[0][i] = make_float4(P.position[0], P.position[1], P.position[2], 0.0f);
            b.dir[0][i] = make_float4(d[0], d[1], d[2], 0.0f);
        }
        b.pathq[0][i] = valid ? i : kNone;
        b.rayq[0][i] = valid ? i | (kKindPrimary << 30) : kNone;
    }
}

// A wave of several sample indices: its finished paths left their samples' values in the slots
// (b.radiance); one thread per pixel adds them to the radiance buffer in sample order (the sums of
// the waves of one sample index, bit for bit), and divides with the last sample. Bound by its reads,
// 16 bytes per sample and 12 written per pixel, coalesced.
__global__ void __launch_bounds__(kWaveThreads)
    wave_resolve_kernel(const WaveView* __restrict__ views, const WaveGen g, const WaveBuffers b)
{
    grid_wait();
    const uint32_t n_views = g.entries / g.samples;
    const uint32_t item = blockIdx.x * kWaveThreads + threadIdx.x;
    const uint32_t per_sample = g.count / g.samples;
    if (item >= per_sample) return;
    const uint32_t bw = g.block_width, bh = 32u / bw;
    uint32_t local;
    const uint32_t vs = __ldg(g.table + wave_entry(g, n_views, item, local));
    const WaveView& V = views[vs & 0xFFFFu];
    const TraceParams& P = V.params;
    if (!V.radiance) return;
    const uint32_t blk = local >> 5, in = local & 31u;
    const uint32_t px = (blk % V.blocks_x) * bw + in % bw;
    const uint32_t py = (blk / V.blocks_x) * bh + in / bw;
    if (px >= P.width || py >= P.height) return;
    const uint32_t first = g.first_sample;
    float* o = V.radiance + 3ull * (py * P.width + px);
    float acc[3] = {0.0f, 0.0f, 0.0f};
    if (first != 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[k] = o[k];
    }
    for (uint32_t s = 0; s < g.samples; ++s) {
        const float4 r = b.radiance[item + s * per_sample];
        acc[0] += r.x;
        acc[1] += r.y;
        acc[2] += r.z;
    }
    const bool last = first + g.samples == P.spp;
#pragma unroll
    for (int k = 0; k < 3; ++k) o[k] = last ? acc[k] / (float)P.spp : acc[k];
}

// The first work of a stage's trace launch: the queues and counters that this stage's other launches
// fill.
__device__ __forceinline__ void begin_stage(const WaveBuffers& b, uint32_t parity)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    for (const uint32_t k : {2 * (parity ^ 1u), 2 * (parity ^ 1u) + 1, kFetchTrace + (parity ^ 1u),  // the next stage's
                             kCountNee, kCountLamp, kFetchLight})                                     // this one's light work
        *counter_of(b, k) = 0;
}

// The rays of a launch. With one view a lane counts its own, and the warp adds them at its end (a launch
// traces either camera rays only or none); with several, one atomic per (view, kind) group of the warp
// at every call (lanes whose rays change views all the time: 6.8 against 5.2 ms on 12 views when each
// lane added its own).
struct RayCounter
{
    bool one_view;
    uint32_t paths = 0, shadows = 0;  // camera or bounce rays; shadow rays
    bool camera = false;
    // Every lane calls; `counted`: it has a ray of `view`.
    __device__ __forceinline__ void add(const WaveView* __restrict__ views, bool counted, uint32_t view, uint32_t kind)
    {
        if (one_view) {
            if (counted && kind == kKindShadow) ++shadows;
            if (counted && kind != kKindShadow) ++paths;
            camera = camera || (counted && kind == kKindPrimary);
            return;
        }
        const uint32_t key = counted ? view * 4u + kind : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        if (counted && (threadIdx.x & 31u) == (uint32_t)__ffs(peers) - 1u) {
            unsigned long long* c = views[view].ray_counts;
            if (c) atomicAdd(c + kind, (unsigned long long)__popc(peers));
        }
    }
    // Every lane calls.
    __device__ __forceinline__ void finish(const WaveView* __restrict__ views)
    {
        if (!one_view) return;
        const bool cam = __any_sync(0xFFFFFFFFu, camera);
        const uint32_t p = __reduce_add_sync(0xFFFFFFFFu, paths), s = __reduce_add_sync(0xFFFFFFFFu, shadows);
        unsigned long long* c = views[0].ray_counts;
        if ((threadIdx.x & 31u) != 0 || !c) return;
        if (p) atomicAdd(c + (cam ? kKindPrimary : kKindBounce), (unsigned long long)p);
        if (s) atomicAdd(c + kKindShadow, (unsigned long long)s);
    }
};

// Ray `i` of the queue (`take`; else none): false for none and for a hole, else its queue entry, view,
// origin, direction and length. Every lane calls.
__device__ __forceinline__ bool next_ray(const WaveView* __restrict__ views, const WaveBuffers& b, uint32_t parity, bool take,
                                         uint32_t i, uint32_t& entry, uint32_t& view, float o[3], float d[3], float& t_max,
                                         RayCounter& counter)
{
    const uint32_t e = take ? b.rayq[parity][i] : kNone;
    const bool ray = e != kNone;
    if (ray) {
        entry = e;
        const uint32_t slot = entry & kSlotMask, kind = entry >> 30;
        view = b.vs[slot] & 0xFFFFu;
        const float4 o4 = b.org[parity][slot];
        const float4 d4 = kind == kKindShadow ? b.sdir[slot] : b.dir[parity][slot];
        o[0] = o4.x;
        o[1] = o4.y;
        o[2] = o4.z;
        d[0] = d4.x;
        d[1] = d4.y;
        d[2] = d4.z;
        t_max = kind == kKindShadow ? d4.w : (kind == kKindPrimary ? kRayTMax : kBounceTMax);
    }
    counter.add(views, ray, view, e >> 30);
    return ray;
}

// The rays that a warp takes at a time: 32, or where the queue fills less than three eighths of the grid's
// lanes 8 or 4 of them in more warps. The lanes of a warp run one after another where their rays differ,
// and these launches last as long as their longest warp. Measured (one B200, 1 spp): 80 x 60 0.182 -> 0.155
// ms, 160 x 90 0.119 -> 0.105, 200 x 150 0.241 -> 0.218, 256 x 200 on 5 k bricks 0.305 -> 0.286, 256 x 256 on 20 k
// 0.382 -> 0.371. With 16 rays from half of the lanes down and 8 from a quarter (in the refilling kernel
// too): 512 x 512 0.424 -> 0.536, the lanes no longer neighbours.
__device__ __forceinline__ uint32_t rays_per_warp(uint32_t n, uint32_t warps)
{
    return n > 12u * warps ? 32u : (n > 4u * warps ? 8u : 4u);
}

__device__ __forceinline__ void write_result(const WaveBuffers& b, uint32_t entry, const Hit& h)
{
    const uint32_t slot = entry & kSlotMask;
    if (entry >> 30 == kKindShadow) b.occluded[slot] = h.hit ? 1u : 0u;
    else b.hit[slot] = h.hit ? make_uint4(__float_as_uint(h.t), h.attrib, h.record, h.group) : make_uint4(0, 0, 0, 0);
}

// The rays of a stage, one per lane from start to end. kEntities: the views' scenes have entities
// (traversed after the world's bricks); the variant without them keeps the world-only DDA's registers.
// Warps take chunks of the queue where there are more than two rays per lane (with entities, whose rays
// differ more, from one on), else a fixed stride.
template <bool kEntities>
__global__ void __launch_bounds__(kWaveThreads)
    wave_trace_kernel(const WaveView* __restrict__ views, const WaveBuffers b, uint32_t parity, bool one_view)
{
    grid_wait();
    const uint32_t n = count_of(b, 2 * parity);
    begin_stage(b, parity);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (kWaveThreads / 32);
    const uint32_t lanes = rays_per_warp(n, warps);
    uint32_t* const fetch = counter_of(b, kFetchTrace + parity);
    RayCounter counter{one_view};
    const bool dynamic = n > 64u * warps || (kEntities && lanes == 32u);
    WarpRange range = {dynamic ? 0u : (blockIdx.x * (kWaveThreads / 32) + threadIdx.x / 32) * lanes, 0};
    const uint32_t chunk = chunk_for(n);
    while (dynamic ? range.more(fetch, n, chunk) : range.at < n) {
        const uint32_t i = lane < lanes ? range.at + lane : n;
        uint32_t entry = 0, view = 0;
        float o[3], d[3], t_max;
        if (next_ray(views, b, parity, i < n, i, entry, view, o, d, t_max, counter)) {
            Hit h;
            if constexpr (kEntities) h = trace_scene_body(views[view].scene, o, d, 0.0f, t_max, entry >> 30 == kKindShadow);
            else h = trace_ray_body(views[view].scene, o, d, 0.0f, t_max);
            write_result(b, entry, h);
        }
        range.at += dynamic ? 32u : warps * lanes;
    }
    counter.finish(views);
}

// The rays after the camera's of a large wave (world bricks only: there is no entity traversal here). They differ widely
// in length: with a ray per lane from start to end 4 of 32 lanes are active on average on a 300 k-brick world. Here a
// lane that has finished waits until kRefill lanes have; these write their results and take the next rays of the
// queue together (7.3 lanes). A lane walks at most kWalkCells empty cells before the lanes that have reached a
// brick test theirs. kRefill of 6 and 20 instead of 12: 1920 x 1080 x 4 spp on 300 k bricks 12.3 and 12.4 against 12.1
// ms; kWalkCells of 3, 8, 64: 12.4, 12.2, 12.8. A pool of 64 rays per warp in shared memory, taken up in phases of
// one kind (10 lanes, but the rays' state through shared memory in every phase): 11.8, but 0.547 against 0.453 for
// 512 x 512. Eight CTAs per SM instead of six: 12.3. Camera rays, whose neighbours walk alike, are faster with a ray
// per lane (1.18 against 1.56 ms for 8.3 M).
//
// Refilling needs a long queue: in the later bounces of a small wave there is nothing to refill from. Frame times with a
// ray per lane over those with refilling (one B200; cubes of 300, 5,000 and 40,000 bricks, terrains of 20,000 and
// 150,000), by paths of the wave:
//   2 bounces:  130 k 0.90 0.97 0.99 0.94 1.01   345 k 0.94 0.99 1.01 1.01 1.04
//   3 bounces:  600 k 0.96 1.02 1.03 0.99 1.06   1 M   0.98 1.03 1.06 1.04 1.09   8 M 1.02 1.09 1.11 1.11 1.16
//   5 bounces:  130 k 0.84 0.89 0.94 0.86 0.91   345 k 0.89 0.94 0.97 0.93 0.98
//   6 bounces:  600 k 0.91 0.97 0.99 0.94 1.00   1 M   0.94 1.02 1.04 1.00 1.06   8 M 1.01 1.09 1.10 1.09 1.15
// The geometric mean over 1, 3 and 6 bounces is 0.985 at 420 k, 0.99 at 600 k and 1.02 at 1 M. Neighbours in a wave of
// several views walk less alike (4 to 8 views, 3 bounces): 164 k 0.96, 200 k 1.02, 369 k 1.03, 400 k 1.05.
constexpr uint32_t kRefill = 12;
constexpr uint32_t kWalkCells = 8;
// Waves of more paths than this are traced so, of one view and of several.
constexpr uint32_t kRefillPaths = 640'000, kRefillPathsViews = 180'000;

__global__ void __launch_bounds__(kWaveThreads, 6)
    wave_trace_refill_kernel(const WaveView* __restrict__ views, const WaveBuffers b, uint32_t parity, bool one_view)
{
    grid_wait();
    const uint32_t n = count_of(b, 2 * parity);
    begin_stage(b, parity);
    uint32_t* const fetch = counter_of(b, kFetchTrace + parity);
    RayCounter counter{one_view};
    WarpRange range = {0, 0};
    const uint32_t chunk = chunk_for(n);
    bool busy = false, done = false, left = true;  // left (warp-uniform): the queue may hold more rays
    uint32_t entry = 0, rec = 0, attrib = 0;       // of a finished ray: attrib 0 is a miss
    float t = 0.0f;
    const SceneView* s = nullptr;
    RayWalk w;
    for (;;) {
        const uint32_t free = __ballot_sync(0xFFFFFFFFu, !busy);
        if (free == 0xFFFFFFFFu || (left && (uint32_t)__popc(free) >= kRefill)) {
            if (done) {
                Hit h;
                h.hit = false;
                if (attrib != 0u) h = walk_hit(*s, w, rec, t, attrib);
                write_result(b, entry, h);
                done = false;
            }
            if (left) left = range.more(fetch, n, chunk);
            if (!left) {
                if (free == 0xFFFFFFFFu) break;
                continue;
            }
            const uint32_t i = range.at + (uint32_t)__popc(free & lanemask_lt());
            const bool take = !busy && i < range.end;
            range.at = min(range.at + (uint32_t)__popc(free), range.end);
            uint32_t view = 0;
            float o[3], d[3], t_max;
            if (next_ray(views, b, parity, take, i, entry, view, o, d, t_max, counter)) {
                s = &views[view].scene;
                busy = walk_begin(*s, o, d, 0.0f, t_max, w);
                done = !busy;
                attrib = 0;
            }
        }
        if (busy) {
            uint2 cell;
            bool at = cell_occupied(s->cells, w.lin, cell);
            for (uint32_t k = 0; k < kWalkCells && !at; ++k) {
                if (!walk_step(w)) {
                    busy = false;
                    break;
                }
                at = cell_occupied(s->cells, w.lin, cell);
            }
            if (busy && at) {
                rec = cell_record(cell, w.lin);
                if (walk_brick(*s, w, rec, 0.0f, t, attrib)) {
                    busy = false;
                } else {
                    attrib = 0;
                    busy = walk_step(w);
                }
            }
            done = !busy;
        }
    }
    counter.finish(views);
}

// kMode: kShadeRender (the render), kShadeRecord (the adjoint's recording pass: also every
// sample's radiance R), kShadeReplay (the adjoint's replay: the gradients, no image).
enum : int
{
    kShadeRender = 0,
    kShadeRecord = 1,
    kShadeReplay = 2,
};

// sum_c G[c] (t[c] s) e[c]: the power gradient of an emission e * P gathered with throughput t and
// weight s (e the material emission without the power).
__device__ __forceinline__ float gsum3(const float G[3], const float t[3], float s, const float e[3])
{
    return G[0] * ((t[0] * s) * e[0]) + G[1] * ((t[1] * s) * e[1]) + G[2] * ((t[2] * s) * e[2]);
}

// The replay's albedo gradients per material code: a CTA sums them in shared memory, in a table of
// kAlbedoCache entries indexed by the code's low bits (the first code to reach an entry owns it; a
// code whose entry another code owns goes to global memory directly), added to the global
// gradients once at the end of the CTA.
constexpr uint32_t kAlbedoCache = 128;
struct AlbedoCache
{
    uint32_t* tag;
    float* sum;
    float* global;
    __device__ __forceinline__ void add(uint32_t code, uint32_t c, float v)
    {
        const uint32_t e = code & (kAlbedoCache - 1u);
        uint32_t owner = tag[e];
        if (owner == kNone) {
            const uint32_t old = atomicCAS(tag + e, kNone, code);
            owner = old == kNone ? code : old;
        }
        if (owner == code) atomicAdd(sum + 3 * e + c, v);
        else atomicAdd(global + 3ull * code + c, v);
    }
};

// The end of a path: its sample's radiance R kept (the recording pass) and its value (a camera ray's
// miss: zero) added to the pixel, or left in its slot for wave_resolve_kernel.
template <int kMode>
__device__ __forceinline__ void finish_path(const WaveView& V, const WaveBuffers& b, const WaveAdjoint& adj, uint32_t slot,
                                            uint32_t item, uint32_t sp, bool zero, const float rad[3], const float e0[3],
                                            const float a0[3], bool resolve)
{
    if (kMode == kShadeReplay) return;
    const TraceParams& P = V.params;
    if (kMode == kShadeRecord) {
        float* rs = adj.sample_radiance + 3ull * ((uint64_t)sp * P.width * P.height + item);
#pragma unroll
        for (int k = 0; k < 3; ++k) rs[k] = zero ? 0.0f : rad[k];
    }
    if (!V.radiance) return;
    float rgb[3] = {0.0f, 0.0f, 0.0f};
    if (!zero) {
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) bad |= isnan(rad[k]) || isinf(rad[k]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float sr = hmin(bad ? 0.0f : rad[k], 65504.0f);
            rgb[k] = e0[k] + a0[k] * sr;
        }
    }
    if (resolve) {
        b.radiance[slot] = make_float4(rgb[0], rgb[1], rgb[2], 0.0f);
    } else {
        float* o = V.radiance + 3ull * item;
        const bool last = sp + 1u == P.spp;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float acc = (sp == 0 ? 0.0f : o[k]) + rgb[k];
            o[k] = last ? acc / (float)P.spp : acc;
        }
    }
}

// A queued hit (four words) of a segment from org along dir.
template <bool kEntities>
__device__ __forceinline__ Hit unpack_hit(const SceneView& S, const uint4 hw, const float org[3], const float dir[3])
{
    Hit h;
    h.hit = true;
    h.t = __uint_as_float(hw.x);
    h.attrib = hw.y;
    h.record = hw.z;
    h.group = hw.w;
    const uint32_t fc = (uint32_t)(__ffs(h.attrib & 0x3Fu) - 1);
    h.normal[0] = fc == 0 ? 1.0f : (fc == 1 ? -1.0f : 0.0f);
    h.normal[1] = fc == 2 ? 1.0f : (fc == 3 ? -1.0f : 0.0f);
    h.normal[2] = fc == 4 ? 1.0f : (fc == 5 ? -1.0f : 0.0f);
#pragma unroll
    for (int k = 0; k < 3; ++k) h.object_hit[k] = org[k] + dir[k] * h.t;
    if constexpr (kEntities) {
        if (h.attrib & kEntityHit) {
            entity_normal(S, h.group >> kEntityShift, h.attrib, h.normal);
            entity_local_hit(S, h.group >> kEntityShift, org, dir, h.t, h.object_hit);
        }
    }
    return h;
}

// The replay's gradients at a hit with emission me * P seen with throughput tp and weight ew: the
// power of the world's brick, and the vertex's albedo from everything gathered after it (R - rad).
__device__ __forceinline__ void replay_vertex(const SceneView& S, const WaveAdjoint& adj, AlbedoCache& cache, const Hit& h,
                                              const float G[3], const float R[3], const float rad[3], const float tp[3],
                                              float ew, const float me[3], const float al[3])
{
    if (!(h.attrib & kEntityHit)) atomicAdd(adj.d_power + h.record, gsum3(G, tp, ew, me));
    const uint32_t code = material_code((h.attrib >> 16) & 0xFFFFu, S.enc);
#pragma unroll
    for (int k = 0; k < 3; ++k)
        if (al[k] > 0.0f && G[k] != 0.0f) cache.add(code, k, G[k] * (R[k] - rad[k]) / al[k]);
}

// kMinBlocks CTAs of 128 threads per SM: 5 (96 registers, no spills) for a scene whose records
// stay in L2, 8 (64 registers; the light kernels spill about 150 bytes) where the descent and the
// record loads go to HBM and more warps in flight hide them (measured: 5 is the fastest of 3 .. 8 on
// the 128^3 world; 8 on the 2 M-brick world and the 64-scene batch).
// kEntities: the views' scenes have entities (their hits, their lights); the variant without
// them keeps the world-only shading's registers. resolve: a finished path leaves its sample in its
// slot for wave_resolve_kernel (several samples of a pixel are in flight).
template <int kMode, int kMinBlocks, bool kEntities>
__global__ void __launch_bounds__(kWaveThreads, kMinBlocks)
    wave_shade_kernel(const WaveView* __restrict__ views, const WaveBuffers b, uint32_t parity, const WaveAdjoint adj,
                      bool resolve, uint32_t first_sample)
{
    grid_wait();
    __shared__ float s_albedo[kMode == kShadeReplay ? kAlbedoCache * 3 : 1];
    __shared__ uint32_t s_tag[kMode == kShadeReplay ? kAlbedoCache : 1];
    AlbedoCache cache{s_tag, s_albedo, adj.d_albedo};
    if (kMode == kShadeReplay) {
        for (uint32_t i = threadIdx.x; i < kAlbedoCache * 3; i += kWaveThreads) s_albedo[i] = 0.0f;
        for (uint32_t i = threadIdx.x; i < kAlbedoCache; i += kWaveThreads) s_tag[i] = kNone;
        __syncthreads();
    }
    const uint32_t n = count_of(b, 2 * parity + 1);
    const uint32_t out = parity ^ 1u;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t stride = gridDim.x * kWaveThreads;
    if (blockIdx.x == 0 && threadIdx.x == 0) *counter_of(b, kFetchShade + out) = 0;  // the next shade launch's
    // Chunks from a fetch counter (as in wave_trace_kernel) for scenes with entities or records that
    // do not stay in L2 (the 8-CTA variants); the fixed stride for the resident scene.
    constexpr bool kDynamic = kEntities || kMinBlocks == 8;
    uint32_t* const fetch = counter_of(b, kFetchShade + parity);
    __shared__ uint32_t s_queue[kWaveThreads / 32][4][kQueueWords];
    uint32_t(*const buffers)[kQueueWords] = s_queue[threadIdx.x >> 5];
    WarpQueue paths = {buffers[0], counter_of(b, 2 * out + 1), b.pathq[out]};
    WarpQueue rays = {buffers[1], counter_of(b, 2 * out), b.rayq[out]};
    WarpQueue draws = {buffers[2], counter_of(b, kCountNee), b.neeq};
    WarpQueue lamps = {buffers[3], counter_of(b, kCountLamp), b.lampq};
    WarpRange range = {kDynamic ? 0u : blockIdx.x * kWaveThreads + (threadIdx.x & ~31u), 0};
    const uint32_t chunk = chunk_for(n);
    for (; kDynamic ? range.more(fetch, n, chunk) : range.at < n; range.at += kDynamic ? 32u : stride) {
        const uint32_t i = range.at + lane;
        uint32_t slot = 0;
        bool live = false, nee = false, lamp = false, ext = false;
        if (i < n) slot = b.pathq[parity][i];
        if (i < n && slot != kNone) {
            const uint32_t f = b.flags[slot];
            const uint32_t vs = b.vs[slot];
            const WaveView& V = views[vs & 0xFFFFu];
            const SceneView& S = V.scene;
            const TraceParams& P = V.params;
            const uint32_t sp = first_sample + (vs >> 16);
            const uint32_t item = b.item[slot];
            const bool primary = (f & kFlagPrimary) != 0;
            float rad[3] = {0.0f, 0.0f, 0.0f};
            if (!primary) {
                const float4 r4 = b.radiance[slot];
                rad[0] = r4.x;
                rad[1] = r4.y;
                rad[2] = r4.z;
            }
            if ((f & kFlagShadow) && !b.occluded[slot]) {
                const float4 s4 = b.sadd[slot];
                rad[0] += s4.x;
                rad[1] += s4.y;
                rad[2] += s4.z;
                if (kMode == kShadeReplay) {
                    const uint2 pn = b.adj_nee[slot];  // the lamp's power gradient, now unoccluded
                    if (pn.x != kNone) atomicAdd(adj.d_power + pn.x, __uint_as_float(pn.y));
                }
            }
            float G[3] = {0.0f, 0.0f, 0.0f}, R[3] = {0.0f, 0.0f, 0.0f};
            if (kMode == kShadeReplay && !primary) {
                const float4 g4 = b.adj_g[slot];
                const float4 r4 = b.adj_r[slot];
                G[0] = g4.x;
                G[1] = g4.y;
                G[2] = g4.z;
                R[0] = r4.x;
                R[1] = r4.y;
                R[2] = r4.z;
            }
            bool finish = true, zero = false;
            float e0[3] = {0.0f, 0.0f, 0.0f}, a0[3] = {0.0f, 0.0f, 0.0f};
            if (!primary) {
                const float4 a4 = b.a0[slot];
                const float4 e4 = b.e0[slot];
                a0[0] = a4.x;
                a0[1] = a4.y;
                a0[2] = a4.z;
                e0[0] = e4.x;
                e0[1] = e4.y;
                e0[2] = e4.z;
            }
            if (f & kFlagExt) {
                const uint4 hw = b.hit[slot];
                if (kMode != kShadeReplay && primary && sp == 0 && P.voxel_id)
                    write_voxel_id<kEntities>(S, P, item, hw.y != 0u, __uint_as_float(hw.x), hw.y, hw.z, hw.w);
                const float4 o4 = b.org[parity][slot];
                const float4 d4 = b.dir[parity][slot];
                const float org[3] = {o4.x, o4.y, o4.z};
                const float dir[3] = {d4.x, d4.y, d4.z};
                if (hw.y == 0u) {
                    zero = primary;  // a missed camera ray: the sample is 0
                } else {
                    const Hit h = unpack_hit<kEntities>(S, hw, org, dir);
                    const uint32_t px = item % P.width, py = item / P.width;
                    const uint32_t seed = P.frame_seed + sp;
                    uint32_t rng;
                    if (primary) rng = init_random(px, py, seed);
                    else rng = b.rng[slot];
                    float tp[3];
                    uint32_t bounce_index, seg_light;
                    float al[3], em[3], o2[3], d2[3];
                    shade<kEntities>(S, h, org, dir, rng, al, em, o2, d2);
                    const uint32_t block = (h.attrib >> 16) & 0xFFFFu;
                    // The replay's power gradients need the material emission without the power.
                    float me[3] = {0.0f, 0.0f, 0.0f};
                    if (kMode == kShadeReplay) {
                        float ma[3];
                        material_of(S, block, ma, me);
                    }
                    bool nee_now;
                    if (primary) {
                        const float t0 = 1.0f / hmax(0.001f, 1.0f);
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            e0[k] = em[k];
                            a0[k] = al[k];
                            rad[k] = 0.0f;
                            tp[k] = t0;
                        }
                        seg_light = 0;
                        bounce_index = 1;
                        nee_now = P.light_nee && P.bounce_count >= 1;
                        if (kMode == kShadeReplay) {
                            // The sample's value e0 + a0 * sanitize(R), R from the recording pass.
                            const float* rs = adj.sample_radiance + 3ull * ((uint64_t)sp * P.width * P.height + item);
                            bool bad = false;
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                R[k] = rs[k];
                                bad |= isnan(R[k]) || isinf(R[k]);
                            }
                            const uint32_t code0 = material_code(block, S.enc);
                            float g[3];
                            bool any = false;
#pragma unroll
                            for (int k = 0; k < 3; ++k) {
                                g[k] = adj.d_radiance[3ull * item + k] / (float)P.spp;
                                const float sr = hmin(bad ? 0.0f : R[k], 65504.0f);
                                cache.add(code0, k, g[k] * sr);
                                G[k] = (!bad && R[k] <= 65504.0f) ? g[k] * a0[k] : 0.0f;
                                any |= G[k] != 0.0f;
                            }
                            if (!(h.attrib & kEntityHit))
                                atomicAdd(adj.d_power + h.record, g[0] * me[0] + g[1] * me[1] + g[2] * me[2]);
                            if (!any) nee_now = false, bounce_index = P.bounce_count + 1u;  // nothing flows back
                        }
                    } else {
                        const float4 t4 = b.throughput[parity][slot];
                        tp[0] = t4.x;
                        tp[1] = t4.y;
                        tp[2] = t4.z;
                        seg_light = (f & kFlagSegLight) ? 3u : 0u;
                        bounce_index = (f & kFlagBounce) + 1u;
                        // A lamp that the segment's light draw could have drawn: its weight, its
                        // emission and the replay's gradients are the light kernel's.
                        lamp = seg_light != 0u && (em[0] > 0.0f || em[1] > 0.0f || em[2] > 0.0f) && !(h.t < kNearField);
                        if (!lamp) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) rad[k] += em[k] * (tp[k] * 1.0f);
                            if (kMode == kShadeReplay) replay_vertex(S, adj, cache, h, G, R, rad, tp, 1.0f, me, al);
                        }
#pragma unroll
                        for (int k = 0; k < 3; ++k) tp[k] *= al[k] / hmax(0.001f, 1.0f);
                        seg_light = 0u;
                        nee_now = P.light_nee && bounce_index <= P.bounce_count;
                    }
                    if (nee_now) {
                        // The draw's shadow contribution carries this vertex's throughput, before
                        // Russian roulette rescales it.
                        seg_light = 3u;
                        nee = true;
                        b.sadd[slot] = make_float4(tp[0], tp[1], tp[2], 0.0f);
                        if (primary) b.light_rng[slot] = init_random(px, py, seed ^ 0x7F4A7C15u);
                    }
                    bool alive = true;
                    if (!primary) {
                        const float cp = hmax(tp[0], hmax(tp[1], tp[2]));
                        alive = !(cp <= 0.0f || cp < random01(rng));
                        if (alive) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) tp[k] *= 1.0f / cp;
                        }
                    }
                    ext = alive && bounce_index <= P.bounce_count;
                    live = nee || ext;
                    finish = !live && !lamp;
                    if (!finish) b.radiance[slot] = make_float4(rad[0], rad[1], rad[2], 0.0f);
                    if (live) {
                        b.flags[slot] = bounce_index | (seg_light ? kFlagSegLight : 0u) | (ext ? kFlagExt : 0u);
                        b.org[out][slot] = make_float4(o2[0], o2[1], o2[2], 0.0f);
                        b.seg_n[out][slot] = make_float4(h.normal[0], h.normal[1], h.normal[2], 0.0f);
                        if (ext) {
                            b.rng[slot] = rng;
                            b.dir[out][slot] = make_float4(d2[0], d2[1], d2[2], 0.0f);
                            b.throughput[out][slot] = make_float4(tp[0], tp[1], tp[2], 0.0f);
                        }
                        if (primary) {
                            b.a0[slot] = make_float4(a0[0], a0[1], a0[2], 0.0f);
                            b.e0[slot] = make_float4(e0[0], e0[1], e0[2], 0.0f);
                            if (kMode == kShadeReplay) {
                                b.adj_g[slot] = make_float4(G[0], G[1], G[2], 0.0f);
                                b.adj_r[slot] = make_float4(R[0], R[1], R[2], 0.0f);
                            }
                        }
                    }
                }
            }
            if (finish) finish_path<kMode>(V, b, adj, slot, item, sp, zero, rad, e0, a0, resolve);
        }
        paths.push(live, slot);
        rays.push(ext, slot | (kKindBounce << 30));
        draws.push(nee, slot);
        lamps.push(lamp, slot | (live ? 0u : kLampEnds));
    }
    paths.finish();
    rays.finish();
    draws.finish();
    lamps.finish();
    if (kMode == kShadeReplay) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kAlbedoCache * 3; i += kWaveThreads) {
            const uint32_t code = s_tag[i / 3];
            if (code != kNone && s_albedo[i] != 0.0f) atomicAdd(adj.d_albedo + 3ull * code + i % 3, s_albedo[i]);
        }
    }
}

// Waves of at most this many paths do their light-tree work with four lanes per item.
constexpr uint32_t kQuadPaths = 1u << 16;

// The next chunk's index for the calling warp, from a fetch counter. Every lane calls.
__device__ __forceinline__ uint32_t fetch_one(uint32_t* counter)
{
    uint32_t c = 0;
    if ((threadIdx.x & 31u) == 0) c = atomicAdd(counter, 1u);
    return __shfl_sync(0xFFFFFFFFu, c, 0);
}

// The light-tree work that the shade launch queued: the light draws (a vertex's NEE up to its shadow
// ray, which is queued), then the lamp hits (the MIS weight of the hit against the draw of the vertex
// before it, then its emission). In the shade kernel, where half of a warp's paths miss or end and
// one in a hundred hits a lamp, these ran with 12 of 32 lanes. Measured against that (one B200): 512 x
// 512, 1 spp 0.520 -> 0.496 ms; 333 x 251, 8 spp 1.11 -> 0.93; 1920 x 1080, 4 spp on 300 k bricks
// 19.9 -> 14.3; the adjoint of 256 x 256, 8 spp over a world of lamps 3.24 -> 2.11. A frame of 14 k
// paths, all launch latency, pays for the third launch per stage: 0.133 -> 0.145.
//
// A warp takes 32 draws or 32 lamp hits, a lane each. kQuad: eight, and four lanes share an item's
// walk through the tree, a child slot each: for waves of few paths, whose launches are chains of
// dependent levels on a chip that is mostly idle. Measured, four lanes against one (1 spp, 4 bounces):
// 200 x 150 0.287 against 0.305 ms, 256 x 256 on 20 k bricks 0.429 against 0.473, 400 x 300 0.376
// against 0.381, 512 x 512 0.578 against 0.516 (there the chip is full, and four lanes repeat the pick).
template <int kMode, int kMinBlocks, bool kEntities, bool kQuad>
__global__ void __launch_bounds__(kWaveThreads, kMinBlocks)
    wave_light_kernel(const WaveView* __restrict__ views, const WaveBuffers b, uint32_t parity, const WaveAdjoint adj,
                      bool resolve, uint32_t first_sample)
{
    grid_wait();
    __shared__ float s_albedo[kMode == kShadeReplay ? kAlbedoCache * 3 : 1];
    __shared__ uint32_t s_tag[kMode == kShadeReplay ? kAlbedoCache : 1];
    AlbedoCache cache{s_tag, s_albedo, adj.d_albedo};
    if (kMode == kShadeReplay) {
        for (uint32_t i = threadIdx.x; i < kAlbedoCache * 3; i += kWaveThreads) s_albedo[i] = 0.0f;
        for (uint32_t i = threadIdx.x; i < kAlbedoCache; i += kWaveThreads) s_tag[i] = kNone;
        __syncthreads();
    }
    const uint32_t draws = count_of(b, kCountNee);
    const uint32_t lamps = count_of(b, kCountLamp);
    constexpr uint32_t chunk = kQuad ? 8u : 32u;
    const uint32_t draw_chunks = (draws + chunk - 1) / chunk;
    const uint32_t chunks = draw_chunks + (lamps + chunk - 1) / chunk;
    const uint32_t out = parity ^ 1u;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* const fetch = counter_of(b, kFetchLight);
    __shared__ uint32_t s_queue[kWaveThreads / 32][kQueueWords];
    WarpQueue rays = {s_queue[threadIdx.x >> 5], counter_of(b, 2 * out), b.rayq[out]};
    for (uint32_t c = fetch_one(fetch); c < chunks; c = fetch_one(fetch)) {
        const bool draw = c < draw_chunks;
        const uint32_t base = (draw ? c : c - draw_chunks) * chunk;
        const uint32_t count = min(chunk, (draw ? draws : lamps) - base);
        const bool mine = lane < count;
        uint32_t slot = 0, entry = 0;
        const SceneView* S = nullptr;
        float x[3] = {0.0f, 0.0f, 0.0f}, nrm[3] = {0.0f, 0.0f, 0.0f};
        bool walk = false;
        const SceneView* set = nullptr;  // the light set the walk is in
        if (draw) {
            LightDraw w = {0u, 0u, 0u, 1.0f};
            uint32_t light_rng = 0;
            if (mine) {
                slot = b.neeq[base + lane];
                S = &views[b.vs[slot] & 0xFFFFu].scene;
                const float4 o4 = b.org[out][slot];
                const float4 n4 = b.seg_n[out][slot];
                x[0] = o4.x;
                x[1] = o4.y;
                x[2] = o4.z;
                nrm[0] = n4.x;
                nrm[1] = n4.y;
                nrm[2] = n4.z;
                light_rng = b.light_rng[slot];
                w.rng = random_u32(light_rng);
                b.light_rng[slot] = light_rng;
                walk = light_tree_pick<kEntities>(*S, x, nrm, w);
                set = (kEntities && w.tree == 1u) ? S->dyn : S;
            }
            uint32_t leaf = kNone;
            if constexpr (!kQuad) {
                if (walk) leaf = light_walk<true>(*set, x, nrm, w);
            } else {
                const uint32_t from = lane >> 2;
                float qx[3], qn[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    qx[k] = __shfl_sync(0xFFFFFFFFu, x[k], from);
                    qn[k] = __shfl_sync(0xFFFFFFFFu, nrm[k], from);
                }
                LightDraw qw;
                qw.rng = __shfl_sync(0xFFFFFFFFu, w.rng, from);
                qw.root = __shfl_sync(0xFFFFFFFFu, w.root, from);
                qw.pdf = __shfl_sync(0xFFFFFFFFu, w.pdf, from);
                const bool busy = __shfl_sync(0xFFFFFFFFu, walk ? 1u : 0u, from) != 0u;
                const uint64_t qset = __shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(set), from);
                const LightBvhNode* nodes = busy ? reinterpret_cast<const SceneView*>(qset)->nodes : nullptr;
                const uint32_t found = light_walk_quad(nodes, busy, qx, qn, qw);
                // Back to the item's lane.
                const uint32_t to = 4u * (lane & 7u);
                const uint32_t l = __shfl_sync(0xFFFFFFFFu, found, to);
                const uint32_t rng = __shfl_sync(0xFFFFFFFFu, qw.rng, to);
                const float pdf = __shfl_sync(0xFFFFFFFFu, qw.pdf, to);
                if (mine) {
                    leaf = l;
                    w.rng = rng;
                    w.pdf = pdf;
                }
            }
            bool shadow = false;
            if (walk) {
                LightPoint p;
                ShadowRay r;
                shadow = light_point(*set, x, w, leaf, p) && nee_shadow_ray<kEntities>(*S, x, nrm, p, r);
                if (shadow) {
                    const float4 t4 = b.sadd[slot];
                    const float tp[3] = {t4.x, t4.y, t4.z};
                    float sadd[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) sadd[k] = r.value[k] * (tp[k] * (1.0f / 1.0f));
                    b.sdir[slot] = make_float4(r.dir[0], r.dir[1], r.dir[2], r.t_max);
                    b.sadd[slot] = make_float4(sadd[0], sadd[1], sadd[2], 0.0f);
                    b.flags[slot] |= kFlagShadow;
                    if (kMode == kShadeReplay) {
                        const float4 g4 = b.adj_g[slot];
                        const float G[3] = {g4.x, g4.y, g4.z};
                        uint2 pending = make_uint2(kNone, 0u);
                        if (r.brick != kNone) {
                            const float gp = G[0] * (tp[0] * r.dvalue_de[0]) + G[1] * (tp[1] * r.dvalue_de[1]) +
                                             G[2] * (tp[2] * r.dvalue_de[2]);
                            pending = make_uint2(r.brick, __float_as_uint(gp));
                        }
                        b.adj_nee[slot] = pending;
                    }
                }
            }
            rays.push(shadow, slot | (kKindShadow << 30));
        } else {
            Hit h;
            LampHit lamp = {nullptr, 0u, kNone, 0.0f};
            float dir[3] = {0.0f, 0.0f, 0.0f};
            bool weighed = false;
            uint32_t vs = 0;
            if (mine) {
                entry = b.lampq[base + lane];
                slot = entry & ~kLampEnds;
                vs = b.vs[slot];
                S = &views[vs & 0xFFFFu].scene;
                const float4 o4 = b.org[parity][slot];
                const float4 d4 = b.dir[parity][slot];
                const float4 n4 = b.seg_n[parity][slot];
                x[0] = o4.x;
                x[1] = o4.y;
                x[2] = o4.z;
                dir[0] = d4.x;
                dir[1] = d4.y;
                dir[2] = d4.z;
                nrm[0] = n4.x;
                nrm[1] = n4.y;
                nrm[2] = n4.z;
                h = unpack_hit<kEntities>(*S, b.hit[slot], x, dir);
                weighed = lamp_lookup(*S, h, x, lamp);
                walk = weighed && lamp.leaf != kNone;
            }
            float probability = 0.0f;
            if constexpr (!kQuad) {
                if (walk) probability = leaf_probability(*S, *lamp.set, lamp.leaf, x, nrm, lamp.tree);
            } else {
                const uint32_t from = lane >> 2;
                float qx[3], qn[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    qx[k] = __shfl_sync(0xFFFFFFFFu, x[k], from);
                    qn[k] = __shfl_sync(0xFFFFFFFFu, nrm[k], from);
                }
                const uint32_t leaf = __shfl_sync(0xFFFFFFFFu, lamp.leaf, from);
                const bool busy = __shfl_sync(0xFFFFFFFFu, walk ? 1u : 0u, from) != 0u;
                const uint64_t qset = __shfl_sync(0xFFFFFFFFu, reinterpret_cast<uint64_t>(lamp.set), from);
                const float found = leaf_walk_quad(reinterpret_cast<const SceneView*>(qset), leaf, busy, qx, qn);
                probability = __shfl_sync(0xFFFFFFFFu, found, 4u * (lane & 7u));
                if (walk) probability = probability * tree_probability(*S, x, nrm, lamp.tree);
            }
            if (mine) {
                const float ew = weighed ? lamp_weight(h, lamp, probability, dir, nrm) : 1.0f;
                const WaveView& V = views[vs & 0xFFFFu];
                const float4 t4 = b.throughput[parity][slot];
                const float4 r4 = b.radiance[slot];
                const float tp[3] = {t4.x, t4.y, t4.z};
                float rad[3] = {r4.x, r4.y, r4.z};
                float al[3], me[3], em[3];
                hit_emission<kEntities>(*S, h, al, me, em);
#pragma unroll
                for (int k = 0; k < 3; ++k) rad[k] += em[k] * (tp[k] * ew);
                if (kMode == kShadeReplay) {
                    const float4 g4 = b.adj_g[slot];
                    const float4 s4 = b.adj_r[slot];
                    const float G[3] = {g4.x, g4.y, g4.z};
                    const float R[3] = {s4.x, s4.y, s4.z};
                    replay_vertex(*S, adj, cache, h, G, R, rad, tp, ew, me, al);
                }
                if (entry & kLampEnds) {
                    const float4 a4 = b.a0[slot];
                    const float4 e4 = b.e0[slot];
                    const float a0[3] = {a4.x, a4.y, a4.z};
                    const float e0[3] = {e4.x, e4.y, e4.z};
                    finish_path<kMode>(V, b, adj, slot, b.item[slot], first_sample + (vs >> 16), false, rad, e0, a0, resolve);
                } else {
                    b.radiance[slot] = make_float4(rad[0], rad[1], rad[2], 0.0f);
                }
            }
        }
    }
    rays.finish();
    if (kMode == kShadeReplay) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kAlbedoCache * 3; i += kWaveThreads) {
            const uint32_t code = s_tag[i / 3];
            if (code != kNone && s_albedo[i] != 0.0f) atomicAdd(adj.d_albedo + 3ull * code + i % 3, s_albedo[i]);
        }
    }
}

}  // namespace

namespace {

// Carves the wave buffers from `base` (null: only the size is wanted); returns the bytes: 280 a slot, and 40
// for the adjoint's arrays where they are wanted.
uint64_t carve(char* base, uint32_t capacity, bool adjoint, WaveBuffers& b)
{
    const uint64_t c = std::max<uint32_t>(capacity, 32);
    uint64_t at = 0;
    const auto take = [&](auto& array, uint64_t count) {
        array = reinterpret_cast<std::remove_reference_t<decltype(array)>>(base + at);
        at += (count * sizeof(*array) + 255u) & ~uint64_t{255};
    };
    b.capacity = capacity;
    take(b.item, c);
    take(b.vs, c);
    take(b.flags, c);
    take(b.rng, c);
    take(b.light_rng, c);
    for (int k = 0; k < 2; ++k) {
        take(b.org[k], c);
        take(b.dir[k], c);
        take(b.throughput[k], c);
        take(b.seg_n[k], c);
        take(b.rayq[k], 2 * c);
        take(b.pathq[k], c);
    }
    take(b.radiance, c);
    take(b.a0, c);
    take(b.e0, c);
    take(b.sdir, c);
    take(b.sadd, c);
    take(b.hit, c);
    take(b.occluded, c);
    take(b.neeq, c);
    take(b.lampq, c);
    take(b.counts, kCountWords);
    if (adjoint) {
        take(b.adj_g, c);
        take(b.adj_r, c);
        take(b.adj_nee, c);
    }
    return at;
}

}  // namespace

uint64_t wave_buffer_bytes(uint32_t capacity, bool adjoint)
{
    WaveBuffers b;
    return carve(nullptr, capacity, adjoint, b);
}

WaveBuffers wave_carve(void* base, uint32_t capacity, bool adjoint)
{
    WaveBuffers b;
    carve(static_cast<char*>(base), capacity, adjoint, b);
    return b;
}

uint32_t WavePlan::largest() const
{
    uint32_t n = 0;
    for (uint32_t i : items) n = std::max(n, i);
    return n;
}

WavePlan wave_plan(const WaveView* views, uint32_t view_count, uint32_t block_width, uint32_t slots)
{
    WavePlan plan;
    plan.one_view = view_count == 1;
    uint32_t max_spp = 0;
    for (uint32_t v = 0; v < view_count; ++v) max_spp = std::max(max_spp, views[v].params.spp);
    const uint32_t bh = 32u / block_width;
    for (uint32_t s = 0; s < max_spp;) {
        // The views that have sample s, their items, and how many sample indices they all have left.
        std::vector<uint32_t> ids, sizes;
        uint64_t items = 0;
        uint32_t bounces = 0, left = max_spp - s;
        for (uint32_t v = 0; v < view_count; ++v) {
            const TraceParams& p = views[v].params;
            if (p.spp <= s) continue;
            const uint64_t bx = (p.width + block_width - 1) / block_width, by = (p.height + bh - 1) / bh;
            ids.push_back(v);
            sizes.push_back((uint32_t)(32ull * bx * by));
            items += 32ull * bx * by;
            bounces = std::max(bounces, p.bounce_count);
            left = std::min(left, p.spp - s);
        }
        uint32_t samples = items ? (uint32_t)std::min<uint64_t>(left, std::max<uint64_t>(slots / items, 1)) : 1u;
        samples = std::min(samples, kWaveMaxSamples);
        plan.first.push_back(s);
        plan.offset.push_back((uint32_t)plan.table.size());
        plan.entries.push_back((uint32_t)ids.size() * samples);
        plan.samples.push_back(samples);
        plan.items.push_back((uint32_t)std::min<uint64_t>(items * samples, 0xFFFFFFFFull));
        plan.bounces.push_back(bounces);
        for (uint32_t k = 0; k < samples; ++k)
            for (uint32_t id : ids) plan.table.push_back(id | (k << 16));
        uint64_t base = 0;
        for (uint32_t k = 0; k < samples; ++k)
            for (uint32_t size : sizes) {
                plan.table.push_back((uint32_t)base);
                base += size;
            }
        s += samples;
    }
    return plan;
}

namespace {

// A chained launch (launch.cuh). Measured against plain ones (one B200): 160 x 90 0.143 -> 0.125 ms,
// 512 x 512 0.488 -> 0.458, the adjoint of 256 x 256, 8 spp 2.00 -> 1.94. With an early trigger, the
// next launch's CTAs waiting on the chip: 0.127, 0.466, 1.94.
template <typename Kernel, typename... Args>
cudaError_t launch(Kernel kernel, uint32_t grid, cudaStream_t stream, Args... args)
{
    return launch_chained(kernel, grid, kWaveThreads, 0, stream, args...);
}

// Every sub-wave of every wave of the plan, its shade kernels in mode kMode with kMinBlocks CTAs
// per SM.
template <int kMode, int kMinBlocks>
cudaError_t wave_run(const WaveView* d_views, const WavePlan& plan, const uint32_t* d_table, const WaveBuffers& b,
                     uint32_t block_width, uint32_t sm_count, const WaveAdjoint& adj, cudaStream_t stream,
                     uint32_t* launches, bool entities = false)
{
    if (b.capacity == 0) return cudaErrorInvalidValue;
    static int trace_blocks[2] = {0, 0}, refill_blocks = 0, shade_blocks[2] = {0, 0}, light_blocks[2] = {0, 0};
    // Asked once; the lock keeps a second thread from reading a half-filled set.
    static std::mutex blocks_mutex;
    static bool blocks_known = false;
    std::unique_lock<std::mutex> blocks_lock(blocks_mutex);
    if (!blocks_known) {
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&trace_blocks[0], wave_trace_kernel<false>,
                                                             kWaveThreads, 0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&trace_blocks[1], wave_trace_kernel<true>, kWaveThreads,
                                                             0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&shade_blocks[0], wave_shade_kernel<kMode, kMinBlocks, false>,
                                                             kWaveThreads, 0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&shade_blocks[1], wave_shade_kernel<kMode, kMinBlocks, true>,
                                                             kWaveThreads, 0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&light_blocks[0], wave_light_kernel<kMode, kMinBlocks, false, false>,
                                                             kWaveThreads, 0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&light_blocks[1], wave_light_kernel<kMode, kMinBlocks, true, false>,
                                                             kWaveThreads, 0));
        CX_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&refill_blocks, wave_trace_refill_kernel, kWaveThreads, 0));
        refill_blocks = std::max(refill_blocks, 1);
        for (int k = 0; k < 2; ++k) {
            light_blocks[k] = std::max(light_blocks[k], 1);
            trace_blocks[k] = std::max(trace_blocks[k], 1);
            shade_blocks[k] = std::max(shade_blocks[k], 1);
        }
        blocks_known = true;
    }
    blocks_lock.unlock();
    uint32_t count = 0;
    for (size_t s = 0; s < plan.items.size(); ++s) {
        // Several sample indices: the whole wave in one sub-wave, then the samples' sums.
        const bool resolve = plan.samples[s] > 1;
        if (resolve && plan.items[s] > b.capacity) return cudaErrorInvalidValue;
        for (uint32_t first = 0; first < plan.items[s]; first += b.capacity) {
            const uint32_t n = std::min(b.capacity, plan.items[s] - first);
            WaveGen g;
            g.table = d_table + plan.offset[s];
            g.entries = plan.entries[s];
            g.first_sample = plan.first[s];
            g.samples = plan.samples[s];
            g.first_item = first;
            g.count = n;
            g.block_width = block_width;
            CX_TRY(cudaMemsetAsync(b.counts, 0, 4 * kCountWords, stream));
            wave_generate_kernel<<<(n + kWaveThreads - 1) / kWaveThreads, kWaveThreads, 0, stream>>>(d_views, g, b);
            ++count;
            // (At least four rays per warp.)
            const uint32_t ray_grid = std::min<uint32_t>((2 * n + kWaveThreads / 8 - 1) / (kWaveThreads / 8),
                                                         sm_count * (uint32_t)trace_blocks[entities ? 1 : 0]);
            const uint32_t shade_grid = std::min<uint32_t>((n + kWaveThreads - 1) / kWaveThreads,
                                                           sm_count * (uint32_t)shade_blocks[entities ? 1 : 0]);
            // At most a light draw and a lamp hit per path; chunks of 32.
            const uint32_t light_grid = std::min<uint32_t>((2 * n + kWaveThreads - 1) / kWaveThreads,
                                                           sm_count * (uint32_t)light_blocks[entities ? 1 : 0]);
            const bool one_view = plan.one_view;
            const bool quad = n <= kQuadPaths;
            const bool refill = !entities && n > (one_view ? kRefillPaths : kRefillPathsViews);
            const uint32_t refill_grid = sm_count * (uint32_t)refill_blocks;
            const uint32_t quad_grid = std::min<uint32_t>((8 * n + kWaveThreads - 1) / kWaveThreads, sm_count * 5);
            const auto stage = [&](auto with_entities, uint32_t it) {
                const uint32_t parity = it & 1u;
                constexpr bool kEntities = decltype(with_entities)::value;
                cudaError_t e = refill && it > 0 ? launch(wave_trace_refill_kernel, refill_grid, stream, d_views, b, parity, one_view)
                                     : launch(wave_trace_kernel<kEntities>, ray_grid, stream, d_views, b, parity, one_view);
                if (e == cudaSuccess)
                    e = launch(wave_shade_kernel<kMode, kMinBlocks, kEntities>, shade_grid, stream, d_views, b, parity, adj,
                               resolve, g.first_sample);
                if (e == cudaSuccess)
                    e = quad ? launch(wave_light_kernel<kMode, 5, kEntities, true>, quad_grid, stream, d_views, b, parity, adj,
                                      resolve, g.first_sample)
                             : launch(wave_light_kernel<kMode, kMinBlocks, kEntities, false>, light_grid, stream, d_views, b,
                                      parity, adj, resolve, g.first_sample);
                return e;
            };
            for (uint32_t it = 0; it <= plan.bounces[s]; ++it) {
                CX_TRY(entities ? stage(std::true_type{}, it) : stage(std::false_type{}, it));
                count += 3;
            }
            if (resolve && kMode != kShadeReplay) {
                CX_TRY(launch(wave_resolve_kernel, (n / g.samples + kWaveThreads - 1) / kWaveThreads, stream, d_views, g, b));
                ++count;
            }
            CX_TRY(cudaGetLastError());
        }
    }
    if (launches) *launches += count;
    return cudaSuccess;
}

}  // namespace

bool wave_resident_scene(const SceneView& s) { return s.brick_count <= kWaveResidentBricks; }

cudaError_t wave_trace(const WaveView* views, const WaveView* d_views, uint32_t view_count, const WavePlan& plan,
                       const uint32_t* d_table, const WaveBuffers& b, uint32_t block_width, uint32_t sm_count,
                       cudaStream_t stream, uint32_t* launches)
{
    const WaveAdjoint none{nullptr, nullptr, nullptr, nullptr};
    bool entities = false;
    for (uint32_t v = 0; v < view_count; ++v) entities |= views[v].scene.entity_count != 0;
    if (view_count == 1 && wave_resident_scene(views[0].scene))
        return wave_run<kShadeRender, 5>(d_views, plan, d_table, b, block_width, sm_count, none, stream, launches,
                                         entities);
    return wave_run<kShadeRender, 8>(d_views, plan, d_table, b, block_width, sm_count, none, stream, launches,
                                     entities);
}

cudaError_t wave_adjoint(const SceneView& scene, const WaveView* d_record, const WaveView* d_replay,
                         const WavePlan& plan, const uint32_t* d_table, const WaveBuffers& b, uint32_t block_width,
                         uint32_t sm_count, const WaveAdjoint& adj, cudaStream_t stream, uint32_t* launches)
{
    const bool entities = scene.entity_count != 0;
    if (wave_resident_scene(scene)) {
        CX_TRY((wave_run<kShadeRecord, 5>(d_record, plan, d_table, b, block_width, sm_count, adj, stream,
                                              launches, entities)));
        return wave_run<kShadeReplay, 5>(d_replay, plan, d_table, b, block_width, sm_count, adj, stream, launches,
                                         entities);
    }
    CX_TRY((wave_run<kShadeRecord, 8>(d_record, plan, d_table, b, block_width, sm_count, adj, stream,
                                          launches, entities)));
    return wave_run<kShadeReplay, 8>(d_replay, plan, d_table, b, block_width, sm_count, adj, stream, launches,
                                     entities);
}

}  // namespace cx
