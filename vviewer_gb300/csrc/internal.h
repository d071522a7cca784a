// Library-internal state behind the C ABI: device buffers, the context and
// scene handles, error helpers, and the pieces of a render shared by the
// one-shot render (api.cu) and the job engine (engine.cu).
#pragma once
#include <atomic>
#include <chrono>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/vvpt.h"
#include "bvh_build.h"
#include "scene_gpu.h"
#include "slot_pool.h"
#include "wavefront.cuh"

namespace vvpt {

// Gives back the path pools of the current device's contexts that no render
// uses; whether that freed memory.
bool reclaim_pools();

struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release()
    {
        if (ptr)
            cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    cudaError_t alloc(size_t n)
    {
        release();
        if (n == 0)
            n = 16;
        cudaError_t e = cudaMalloc(&ptr, n);
        if (e == cudaErrorMemoryAllocation && reclaim_pools()) {
            cudaGetLastError();
            e = cudaMalloc(&ptr, n);
        }
        if (e == cudaSuccess)
            bytes = n;
        else
            ptr = nullptr;
        return e;
    }
    void swap(DevBuf &o)
    {
        std::swap(ptr, o.ptr);
        std::swap(bytes, o.bytes);
    }
    // grow-only reuse
    cudaError_t reserve(size_t n)
    {
        if (ptr && bytes >= n)
            return cudaSuccess;
        return alloc(n);
    }
    template <class T>
    T *as() const
    {
        return reinterpret_cast<T *>(ptr);
    }
};

struct DeviceMem {
    static void *alloc(size_t n)
    {
        void *p = nullptr;
        if (cudaMalloc(&p, n) == cudaSuccess)
            return p;
        cudaGetLastError();
        return nullptr;
    }
    static void *alloc_or_reclaim(size_t n)
    {
        void *p = alloc(n);
        return p || !reclaim_pools() ? p : alloc(n);
    }
    static void free(void *p) { cudaFree(p); }
    static size_t free_bytes()
    {
        size_t free = 0, total = 0;
        if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return free;
    }
};

struct Engine; // engine.cu

// Meshes built and packed on the device (bvh_gpu.cu): the first part of the
// scene's node, triangle, vertex and index arrays. Each mesh's links are
// relative to its root node.
struct DeviceMeshes {
    struct Placed {
        uint32_t node_offset = 0, tri_offset = 0, vertex_offset = 0; // its index triples start at tri_offset too
        Box3 root{};
    };
    std::vector<Placed> placed;                 // per mesh, in the order given
    std::vector<std::unique_ptr<DevBuf>> nodes; // in order, num_nodes in all
    // the scene's arrays themselves: behind the device's part there is room for
    // `host_tris`, `host_verts` and `host_index_tris` more elements
    DevBuf tris, verts, indices;
    uint64_t host_tris = 0, host_verts = 0, host_index_tris = 0;
    uint32_t num_nodes = 0, num_tris = 0, num_verts = 0;
    int depth = 0;
    bool no_room = false; // an allocation failed for lack of memory

    void release()
    {
        nodes.clear();
        for (DevBuf *b : {&tris, &verts, &indices})
            b->release();
        num_nodes = num_tris = num_verts = 0;
    }
};
bool build_meshes_gpu(const vvpt_scene_desc *desc, const std::vector<uint32_t> &meshes, const BVHBuildOptions &opt,
                      cudaStream_t stream, DeviceMeshes &out, std::string &err);

}  // namespace vvpt

struct vvpt_scene {
    vvpt::DevBuf nodes, wnodes, tris, verts, indices, instances, tlas_order, materials, lights, textures, texels, env_dist,
        emit_boxes;
    vvpt::SceneView view{};
    uint64_t bytes = 0;
    uint32_t num_materials = 0;
    std::atomic<uint32_t> jobs_in_flight{0}; // engine jobs that still read this scene
};

struct vvpt_ctx {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    std::mutex mu;
    std::string last_error;
    std::atomic<float> progress{0.0f};
    vvpt_render_stats stats{};
    vvpt_tuning tuning{};
    // render buffers (grow-only, reused across renders)
    vvpt::SlotPool<vvpt::DeviceMem> pool;
    vvpt::DevBuf results, params, outputs;
    uint32_t *counters_pinned = nullptr;
    vvpt::DevBuf rays, hits, err_word;
    cudaStream_t user_stream = nullptr;
    vvpt_kernel_profile profile{};
    // job engine (vvpt_submit ...), created on first use
    std::mutex engine_mu;
    vvpt::Engine *engine = nullptr;
    std::atomic<uint64_t> budget_bytes{0}; // 0: no limit beyond the device's memory
    int bvh_builder = 0;       // VVPT_BVH_BUILDER_*
    // low-discrepancy sampler tables (VVPT_RENDER_SAMPLER_PMJ), uploaded on first use
    std::mutex sampler_mu;
    vvpt::DevBuf pmj_table, blue_noise_table;
    std::chrono::steady_clock::time_point created = std::chrono::steady_clock::now();
};

namespace vvpt {

inline cudaStream_t vv_stream(const vvpt_ctx *ctx) { return ctx->user_stream ? ctx->user_stream : ctx->stream; }

inline vvpt_status fail(vvpt_ctx *ctx, vvpt_status code, const std::string &msg)
{
    if (ctx)
        ctx->last_error = msg;
    return code;
}

inline vvpt_status cuda_fail(vvpt_ctx *ctx, cudaError_t e, const char *what)
{
    cudaGetLastError();
    std::string m = std::string(what) + ": " + cudaGetErrorString(e);
    return fail(ctx, e == cudaErrorMemoryAllocation ? VVPT_ERR_OOM : VVPT_ERR_DEVICE, m);
}

#define VV_CUDA(call, what)                  \
    do {                                     \
        cudaError_t _e = (call);             \
        if (_e != cudaSuccess)               \
            return cuda_fail(ctx, _e, what); \
    } while (0)

// RenderParams of one render request (SceneData and RenderInfo of the
// reference: VulkanRendererPathTracing.cpp:143-199, raygen.rgen.glsl:24-40).
// Checks the request; on error sets ctx's message and returns its status.
vvpt_status make_render_params(vvpt_ctx *ctx, const vvpt_scene *scene, const vvpt_scene_data *sd,
                               const vvpt_render_info *info, RenderParams &hp);

// The queues of `slots` paths (queue_bytes) in one allocation.
Queues carve_queues(char *base, size_t slots);

// Engine teardown (vvpt_destroy): stops the worker, fails unfinished jobs.
void engine_shutdown(vvpt_ctx *ctx);

}  // namespace vvpt
