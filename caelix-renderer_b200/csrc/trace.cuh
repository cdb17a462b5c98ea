// The trace kernel's launch interface (trace.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "scene.cuh"

namespace cx {

// One render call: the pinhole camera (caelix.h CaelixCamera, without jitter) and the lighting
// options of the path tracer.
struct TraceParams
{
    float position[3];
    float right[3];
    float up[3];
    float forward[3];
    float tan_half_fov_y;
    float aspect;
    uint32_t width;
    uint32_t height;
    uint32_t spp;           // samples per pixel: frame seeds frame_seed .. frame_seed + spp - 1, averaged
    uint32_t bounce_count;  // stochastic bounces after the primary hit
    uint32_t frame_seed;
    uint32_t light_nee;  // 1: light-tree NEE with MIS
    uint32_t* voxel_id;   // optional: width * height uint2, the camera ray's first hit (first sample)
    float voxel_id_tmax;  // hits farther than this are misses of the voxel id (0: no limit)
};

// radiance: width * height fp32 RGB; ray_counts (may be null): u64 primary, bounce, shadow rays,
// accumulated.
cudaError_t trace_launch(const SceneView& s, const TraceParams& p, float* radiance, unsigned long long* ray_counts,
                         cudaStream_t stream);

// The adjoint of a frame (backward.cu): d_radiance = dL/d(radiance), width * height RGB;
// d_albedo (kMaterialCodes x 3, per material code) and d_power (one per brick, the scene's order) are accumulated
// into (zero them first); image (may be null) receives the forward radiance; ray_counts (may be
// null) the rays of the recording pass. `memory`: adjoint_bytes(p, wave_capacity) bytes of device
// memory, 256-aligned (wave_capacity 0 = a path for every item of the largest wave; merge_slots:
// the wave plan's `slots`, wave_merge_slots(wave_capacity) or 0 for one sample index per wave).
uint64_t adjoint_bytes(const TraceParams& p, uint32_t wave_capacity, uint32_t merge_slots);
cudaError_t adjoint_launch(const SceneView& s, const TraceParams& p, const float* d_radiance, float* image,
                           float* d_albedo, float* d_power, unsigned long long* ray_counts, void* memory,
                           uint32_t wave_capacity, uint32_t merge_slots, uint32_t sm_count, cudaStream_t stream,
                           uint32_t* launches);

// ---- the wavefront trace (wave.cu) ----
//
// Paths live in HBM (structure of arrays, one slot per path); a wave is every pixel of one or more
// consecutive sample indices of the views that have them (WavePlan), a wave of one sample index
// split into sub-waves of at most `capacity` slots. Per bounce
// three kernels run over compacted queues: wave_trace_kernel traces every queued ray (extension
// and shadow rays alike, one DDA code path), wave_shade_kernel advances every live path by one
// vertex (shadow result, emission, albedo, Russian roulette) and queues its extension ray and its
// light-tree work, and wave_light_kernel does that work: the light draws (queueing the shadow rays)
// and the MIS weights of lamp hits. Each kernel is small, and its warps start full.

struct WaveView
{
    SceneView scene;
    TraceParams params;
    float* radiance;                 // width * height fp32 RGB (accumulated over the samples)
    unsigned long long* ray_counts;  // u64 primary, bounce, shadow rays of this view
    uint32_t blocks_x;               // pixel blocks per row (block_width x 32 / block_width pixels)
    uint32_t pad;
};

struct WaveBuffers
{
    uint32_t capacity = 0;  // slots
    uint32_t* item = nullptr;   // pixel index within the view (y * width + x)
    uint32_t* vs = nullptr;     // view | sample of the wave << 16
    uint32_t* flags = nullptr;
    uint32_t* rng = nullptr;
    uint32_t* light_rng = nullptr;
    // The segment of a stage's parity (wave_shade_kernel writes the next one's; wave_light_kernel
    // reads both): origin (the shadow ray's too), direction, throughput, the normal it left.
    float4* org[2] = {nullptr, nullptr};
    float4* dir[2] = {nullptr, nullptr};
    float4* throughput[2] = {nullptr, nullptr};
    float4* seg_n[2] = {nullptr, nullptr};
    float4* radiance = nullptr;
    float4* a0 = nullptr;    // primary albedo
    float4* e0 = nullptr;    // primary emission
    float4* sdir = nullptr;  // pending shadow ray: direction, t_max
    float4* sadd = nullptr;  // a light draw's vertex throughput, then the pending shadow contribution
    uint4* hit = nullptr;    // t bits, attrib (0 = miss), record, group
    uint32_t* occluded = nullptr;
    uint32_t* rayq[2] = {nullptr, nullptr};   // 2 * capacity entries: slot | kind << 30
    uint32_t* pathq[2] = {nullptr, nullptr};  // capacity entries
    uint32_t* neeq = nullptr;                 // capacity entries: slots that draw a light
    uint32_t* lampq = nullptr;                // capacity entries: slots whose hit is a lamp (bit 31: the path ends there)
    uint32_t* counts = nullptr;               // queue lengths and fetch counters (wave.cu)
    // The adjoint's per-slot state (wave_adjoint): dL/dR of the sample, its radiance R, the power
    // gradient of a pending NEE lamp (brick, value; applied if its shadow ray is unoccluded).
    float4* adj_g = nullptr;
    float4* adj_r = nullptr;
    uint2* adj_nee = nullptr;
};

// The arrays of an adjoint (wave_adjoint, one view): dL/d(pixel), the radiance of every pixel
// sample (spp x width x height x 3, written by the recording pass, read by the replay), and the
// gradients (accumulated into).
struct WaveAdjoint
{
    const float* d_radiance;
    float* sample_radiance;
    float* d_albedo;  // [kMaterialCodes][3]
    float* d_power;   // [brick_count]
};

// adjoint: with the adjoint's arrays (wave_adjoint; a plain render has none).
uint64_t wave_buffer_bytes(uint32_t capacity, bool adjoint = false);
WaveBuffers wave_carve(void* base, uint32_t capacity, bool adjoint = false);

// The wave plan of a set of views. A wave holds the samples [first, first + samples) of the views
// with spp > first (every one of them has all these samples): its entries are (view, sample) pairs,
// sample by sample, each with its first item (pixel blocks x 32 per entry). More than one sample
// index joins a wave while its items fit `slots` (they are then all in flight at once); a wave of
// one sample index may be larger.
//
// A wave of few paths leaves the chip idle: a launch lasts as long as its longest ray, and one
// sample of a 256 x 256 frame is 65,536 paths on 148 SMs. Measured (one B200), one wave per sample
// index against several in one wave: 333 x 251, 8 spp 3.65 against 1.48 ms; the adjoint of 256 x 256,
// 8 spp 7.60 against 3.83 ms; 1920 x 1080, 4 spp (8.3 M paths at once) 25.5 against 20.4 ms. Fewer
// slots: 1.78 ms for the first at 512 k (two waves), 25.2-27.1 ms for the last at 1 M and 2 M (it
// then runs one sample at a time). At 2^23 slots the path state is 2.35 GB (2.68 with the adjoint's), of 180.
struct WavePlan
{
    std::vector<uint32_t> table;     // per wave: entries (view | sample of the wave << 16), then item bases
    std::vector<uint32_t> first;     // per wave: its first sample index
    std::vector<uint32_t> offset;    // per wave: first word of its entries in `table`
    std::vector<uint32_t> entries;   // per wave: number of entries
    std::vector<uint32_t> samples;   // per wave: sample indices
    std::vector<uint32_t> items;     // per wave: items
    std::vector<uint32_t> bounces;   // per wave: the largest bounce count of its views
    bool one_view = false;
    uint32_t largest() const;        // the items of the largest wave
};
constexpr uint32_t kWaveMergeSlots = 1u << 23;
constexpr uint32_t kWaveMaxSamples = 1u << 16;  // of a wave: an entry's sample has 16 bits
WavePlan wave_plan(const WaveView* views, uint32_t view_count, uint32_t block_width, uint32_t slots);
// The plan's `slots` for a single view's render or adjoint with a wave capacity (0: not set).
inline uint32_t wave_merge_slots(uint32_t wave_capacity)
{
    return wave_capacity && wave_capacity < kWaveMergeSlots ? wave_capacity : kWaveMergeSlots;
}

// Records the trace of every sample of every view into `stream` (no host synchronisation):
// d_views the device copy of `views`, d_table the device copy of plan.table. The views'
// radiance buffers receive the averaged radiance (the per-frame kernel's result, bit for bit).
// Kernel launches recorded are added to *launches (may be null).
// A single view of a scene of at most kWaveResidentBricks bricks (records about 72 MB: they stay
// in the 126 MB L2) runs the shade kernels at 5 CTAs per SM, anything larger or a batch at 8.
constexpr uint32_t kWaveResidentBricks = 65536;
cudaError_t wave_trace(const WaveView* views, const WaveView* d_views, uint32_t view_count, const WavePlan& plan,
                       const uint32_t* d_table, const WaveBuffers& b, uint32_t block_width, uint32_t sm_count,
                       cudaStream_t stream, uint32_t* launches);

// The adjoint of wave_trace for one view (path replay, sampling held fixed; backward.cu states the
// estimator and its derivative): a recording pass (the trace of d_record: radiance into its
// radiance buffer when not null, every sample's R into adj.sample_radiance), then the replay of
// every path (d_replay: the same view without radiance buffer or ray counters) gathering dL/dalbedo
// and dL/dpower. Gradients are accumulated into (zero them first).
cudaError_t wave_adjoint(const SceneView& scene, const WaveView* d_record, const WaveView* d_replay,
                         const WavePlan& plan, const uint32_t* d_table, const WaveBuffers& b, uint32_t block_width,
                         uint32_t sm_count, const WaveAdjoint& adj, cudaStream_t stream, uint32_t* launches);

// ---- the batched persistent trace (trace_batch.cu) ----

constexpr uint32_t kMaxBatchViews = 256;  // views of one persistent launch
constexpr uint32_t kBatchThreads = 128;

// One viewport of a batch, device-resident: its scene, camera and options, output and counters.
// Work items are pixels: item_base + 32 * block + lane, blocks of block_width x (32 / block_width)
// pixels in row-major order over the viewport (blocks_x per row).
struct BatchView
{
    SceneView scene;
    TraceParams params;
    float* radiance;                  // width * height fp32 RGB
    unsigned long long* ray_counts;   // u64 primary, bounce, shadow rays of this view, accumulated
    uint32_t item_base;
    uint32_t blocks_x;
};

struct BatchLaunch
{
    const BatchView* views;
    uint32_t view_count;     // <= kMaxBatchViews
    uint32_t item_count;     // total work items of the views
    uint32_t block_width;    // 8, 16 or 32
    uint32_t refill_min;     // a warp takes new pixels once this many of its lanes are idle (1..32)
    uint32_t* next_item;     // the work counter, zero before the launch
};

// The register-cap variants of the persistent kernel: `min_blocks` CTAs of 128 threads resident
// per SM (4: 128 registers, 6: 80, 8: 64).
bool trace_batch_variant_ok(uint32_t min_blocks);
// Resident CTAs per SM of a variant (the occupancy calculator), 0 for an unknown variant.
int trace_batch_blocks_per_sm(uint32_t min_blocks);
cudaError_t trace_batch_launch(const BatchLaunch& launch, uint32_t min_blocks, uint32_t grid, cudaStream_t stream);

}  // namespace cx
