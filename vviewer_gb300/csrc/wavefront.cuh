// Wavefront path-tracer state and launch interface.
#pragma once
#include <algorithm>

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/vvpt.h"
#include "scene_gpu.h"

namespace vvpt {

// Per-render constants (SceneData + PathTracingData of the reference,
// src/lib/vengine/core/Scene.hpp:27-35 and
// src/lib/vengine/vulkan/renderers/VulkanRendererPathTracing.hpp:57-61).
struct RenderParams {
    float4 view_inv[4]; // columns
    float4 proj_inv[4]; // columns
    float3 background;
    float env_type;     // background.a: 0 solid, 1 HDRI, 2 solid + HDRI lighting
    float lens_radius;
    float focal_distance;
    float env_intensity;
    float zfar;          // sceneData.volumes.b
    float zfar_trunc;    // float(uint(zfar)), rayPrimary.rmiss.glsl:49
    int32_t cam_volume;  // sceneData.volumes.r (-1: camera not in a medium)
    uint32_t width, height;
    uint32_t batch_size, batches, depth, total_samples;
    uint32_t num_lights;  // pathTracingData.lights.r
    uint32_t total_items; // width * height * batches
    uint32_t want_m2;
    uint32_t reduce_fp64; // 1: batch sums added in double (VVPT_RENDER_REDUCE_FP64)
    uint32_t env_light;   // 1: the environment is sampled as one more light (VVPT_RENDER_ENV_IS)
    uint32_t sampler;     // 0: RTGEMS stream, 1: PMJ (VVPT_RENDER_SAMPLER_PMJ)
    const float *pmj;        // [16][16384][2] (sampler 1)
    const float *blue_noise; // [48][128][128] (sampler 1)
};

// Path state of one slot. A slot runs one (pixel, batch) work item: its
// batch_size samples in order, because the RTGEMS state carries from one sample
// to the next (raygen.rgen.glsl:36-55).
// The queues hold slots in the order in which atomics handed out their places,
// so a warp's 32 slots lie all over the pool. What a kernel touches of a slot
// costs whole 32-byte sectors: members that are used together share one, and a
// lane reads or writes both with one 32-byte access. What it touches in memory
// costs more again where it is spread over more lines: tracing and shading keep
// to the first 128 bytes, regeneration mostly to the second.
// (1080p x 32 medium scene, an array per member: shading 74 ms, regeneration 26,
// a render 255; an array per pair of members: 57, 15 and 225; with more slots
// 54, 14.6 and 170; records: 48, 14.2 and 164. The sky scene, whose paths stay
// in order for longer, 47.9 and 48.5.)
struct alignas(128) PathRecord {
    float4 hit; // t, u, v, prim bits
    union {
        struct {
            uint32_t flags, vol;
            uint32_t job; // index into the job table
            uint32_t hit_inst;
        };
        uint4 meta; // the four in one access
    };
    float4 o, d;   // ray origin, direction (xyz)
    float4 beta;   // throughput (xyz), sampler state (w bits)
    float4 rad;    // sample radiance (xyz)
    float4 sh_dir; // shadow direction (xyz), tmax (w)
    float4 sh_c;   // unoccluded light contribution (xyz)
    float4 nee_b;  // beta for the emitter-ray contribution (xyz), BSDF pdf (w)
    float4 nee_c;  // emitter-ray contribution of a path flagged F_NEE (xyz), added by regen or shade
    // first hit, carried across samples (payload semantics)
    float4 alb, nrm;
    // per-batch sums (cumRadiance/cumAlbedo/cumNormal), and in two of their w:
    // work item within its job (batch * width * height + pixel), sample
    float4 cum_rad, cum_alb, cum_nrm;
    float4 unused;
};
static_assert(sizeof(PathRecord) == 256, "path record");

struct PathState {
    PathRecord *slots;
#ifdef __CUDACC__
    __device__ __forceinline__ PathRecord &operator[](uint32_t slot) const { return slots[slot]; }
#endif
};

enum CounterIndex {
    C_EXT0 = 0,
    C_EXT1 = 1,
    C_SHADE_L = 2,
    C_SHADE_P = 3,
    C_SHADE_M = 4,
    C_CONN = 5,
    C_REGEN0 = 6,
    C_REGEN1 = 7,
    C_NEXT_ITEM = 8,
    C_ACTIVE = 9,
    C_ERR = 10,
    C_SEGMENTS = 11,
    C_SHADOW = 12,
    C_NEE = 13,
    C_PATHS = 14,
    C_WALK = 15,
    C_NEEQ = 16,
    C_FETCH = 17,   // rays k_trace has handed out so far in this iteration (lane refill)
    C_NEE_RUN = 18, // emitter rays of this iteration's k_walk (C_NEEQ counts the next one's)
    C_COUNT = 19
};

struct Queues {
    uint32_t *ext[2];
    uint32_t *ext_key;  // per extension-queue entry: shade bin (0 Lambert, 1 PBR, 2 miss) | 4 = emitter walk
    uint32_t *shade_l, *shade_p, *shade_m;
    uint32_t *walk;     // paths whose shadow ray or fused emitter ray needs the full candidate walk
    uint32_t *conn;     // paths with a shadow ray (traced with the next iteration's extension rays)
    uint32_t *nee;      // paths that end with an emitter ray (next iteration's k_walk)
    uint32_t *regen[2];
    uint32_t *counters; // CounterIndex
};

// Per-(pixel, batch) sums written when a work item finishes, reduced in batch
// order at the end so the image equals the reference's per-batch
// read-modify-write sequence (raygen.rgen.glsl:134-144).
struct BatchResults {
    float4 *rad;
    float4 *alb;
    float4 *nrm;
};

// One render job: its scene, its parameters and its per-batch sums. The
// table holds one per job slot; a slot is reused once its job has finished.
struct JobView {
    SceneView scene;
    RenderParams params;
    BatchResults results;
};

// Work items of all admitted jobs form one global sequence, handed out in
// admission order: global item range_begin[r] + i is work item i of job slot
// range_job[r] (ranges ascending). Fused per stage, every queue holds paths of
// all live jobs; a path finds its job through ps.job.
struct JobTable {
    const JobView *jobs;                   // per job slot
    const JobView *only = nullptr;         // host copy of the table's one job (a render), or null
    const unsigned long long *range_begin; // per hand-out range, ascending
    const uint32_t *range_job;
    uint32_t *item_done;                   // per job slot: work items finished
    unsigned long long *next_item;         // next global work item to hand out
    unsigned long long *total_items;       // end of the last range
    uint32_t *num_ranges;
    uint32_t *idle;                        // slots that found no work
    uint32_t *idle_count;
};

struct LaunchShape {
    int grid;
    int block;
    int num_sms;
    uint32_t slots; // path slots: the most entries a queue can hold
    bool automatic; // `grid` is the default, not a caller's blocks_per_sm
};

// Grid of a kernel: at most `grid` blocks, and none past what the slots can
// occupy (`per_block` each): they would only cost their launch, since the loops
// stride over the grid. The default shape also stays within what fits at once,
// `per_sm` blocks of 256 threads; a caller's number reaches every kernel.
inline int launch_blocks(const LaunchShape &shape, int grid, int per_sm, uint32_t per_block)
{
    const uint64_t full = ((uint64_t)shape.slots + per_block - 1) / per_block;
    uint64_t n = std::min<uint64_t>((uint64_t)grid, full);
    if (shape.automatic)
        n = std::min(n, (uint64_t)shape.num_sms * per_sm * 256 / shape.block);
    return (int)std::max<uint64_t>(1, n);
}

// Kernel launchers (wavefront.cu). Each reads its work count from `counters`,
// so a sequence of them can be captured in a CUDA graph.
void launch_iteration(const JobTable &jt, const PathState &ps, const Queues &q, int pingpong, const LaunchShape &shape,
                      cudaStream_t stream);
void launch_reduce(const RenderParams &hparams, const BatchResults &br, float4 *radiance, float4 *albedo,
                   float4 *normal, float4 *radiance_m2, cudaStream_t stream);
// Resets counters, the job table counters and puts every slot on the first
// regeneration queue (its flags cleared).
void launch_init_slots(const Queues &q, const PathState &ps, const JobTable &jt, uint32_t slots, cudaStream_t stream);
// Admits work: raises the global item count to `total_items` over
// `num_ranges` hand-out ranges (after work items ran out, the hand-out counter
// is brought back to the old total) and returns idle slots to the first
// regeneration queue. Launched between graph replays, stream-ordered, after
// the range arrays were written.
void launch_admit(const Queues &q, const JobTable &jt, unsigned long long total_items, uint32_t num_ranges,
                  cudaStream_t stream);
// `status`: error bits and a hand-out counter, both zero before the launch.
void launch_trace_closest(const SceneView &s, const float4 *rays, uint32_t n, vvpt_hit *hits, uint32_t *status,
                          int num_sms, cudaStream_t stream);
// One wavefront kernel, launched on its own (profiling mode); an iteration
// launches all of them in this order.
enum KernelId {
    K_REGEN = 0,
    K_TRACE = 1, // extension rays, then the shadow rays of the previous shading
    K_PARTITION = 2,
    K_WALK = 3, // candidate walks, then the emitter rays of paths that ended
    K_SHADE = 4,
    K_NUM = 5
};
// K_SHADE launches one kernel over the three material-sorted queues, or with
// VVPT_SHADE_SPLIT = 1 (a build option) one kernel per queue, each compiled
// for its own surface model. Measured on the 1080p medium scene: the same
// shading time either way (the split kernels need the same 128 registers,
// set by the medium, light-sampling and emitter-ray code they share; capped
// at 3 blocks per SM they spill and run slower), so one launch.
#ifndef VVPT_SHADE_SPLIT
#define VVPT_SHADE_SPLIT 0
#endif
constexpr int kShadeLaunches = VVPT_SHADE_SPLIT ? 3 : 1;
constexpr int launches_of(int k) { return k == K_SHADE ? kShadeLaunches : 1; }
constexpr int kKernelsPerIteration = K_NUM + kShadeLaunches - 1;
void launch_kernel(KernelId k, const JobTable &jt, const PathState &ps, const Queues &q, int pingpong,
                   const LaunchShape &shape, cudaStream_t stream);

// Algorithmic bytes per work unit of each kernel: the path-state, queue and
// hit-record loads and stores the kernel's code performs for one queue entry
// (nominal branch), plus the three shading vertices and their indices read by
// shade. BVH nodes, triangles and textures are excluded.
constexpr double kBytesPair = 2 * sizeof(float4); // two members in one access
constexpr double kBytesRegen = 4 + 16 /* meta */ + 3 * kBytesPair + sizeof(float4) /* beta rad alb nrm sums */ + 16 +
                               3 * kBytesPair + sizeof(float4) /* writes */ + 4;
// an extension ray's or a shadow ray's entry (the larger of the two, a visible light's)
constexpr double kBytesTrace = 4 + 16 /* meta */ + kBytesPair /* o d */ + sizeof(float4) /* sh_dir */ +
                               3 * sizeof(float4) /* rad sh_c, rad */;
constexpr double kBytesPartition = 4 + 4 + 4;
constexpr double kBytesWalk = 4 + 4 + 4 + 4 * sizeof(float4) /* o d nee_b rad */ + sizeof(float4) + 4;
constexpr double kBytesShade = 4 + 3 * kBytesPair /* hit meta, beta rad, o d */ + 3 * 4 +
                               3 * sizeof(ShadeVertex) /* vertices */ + 2 * 4 + 2 * kBytesPair /* writes */ +
                               2 * kBytesPair + sizeof(float4) /* alb nrm, sh_dir sh_c, nee_b */ +
                               sizeof(float4) /* nee_b read */ + 2 * 4;

}  // namespace vvpt
