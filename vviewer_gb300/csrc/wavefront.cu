// Wavefront integrator kernels: regen (camera rays), trace (closest hits of
// the extension rays and the shadow rays of the previous shading), partition,
// walk (the rays that need the full any-hit candidate walk) and shade
// (surface / medium / miss events, light and BSDF sampling, Russian roulette).
//
// One iteration of the kernels advances every live path by one traced
// segment, i.e. one pass of the `for d < depth` loop of
// src/lib/vengine/shaders/pt/raygen.rgen.glsl:100-124 with the closest-hit /
// miss shader that follows it. The shadow and emitter rays the reference
// traces inside its hit shaders (lightSampling.glsl:108-144,
// next_event_estimation.glsl:1-33) are traced with the next iteration's
// extension rays; they consume no random numbers, so the RNG stream per path
// is the reference's.
#include "shade.cuh"
#include "traverse.cuh"
#include "wavefront.cuh"

namespace vvpt {

// path flag bits
constexpr uint32_t F_SAMPLED = 128u;     // ray direction sampled (BSDF or phase), pdf in nee_b.w
constexpr uint32_t F_INSIDE = 1u;       // rayPayloadPrimary.insideVolume
constexpr uint32_t F_DONE = 2u;         // sample finished, finalize in regen
constexpr uint32_t F_ITEM = 4u;         // slot holds a work item
constexpr uint32_t F_SHADOW = 8u;       // pending shadow connection
constexpr uint32_t F_NEE = 16u;         // pending emitter connection (traced on its own, result in nee_c)
constexpr uint32_t F_NEE_FUSED = 32u;   // emitter ray rides on the next extension ray
constexpr uint32_t F_NEE_FULL = 64u;    // ... but needs the full candidate walk (set by k_partition)
constexpr uint32_t F_SHADOW_WALK = 1u << 24; // shadow ray needs the candidate walk (set by k_trace)
constexpr int kDepthShift = 8;          // recursionDepth d
constexpr int kSurfShift = 16;          // surfaceDepth
constexpr uint32_t kByteMask = 0xFFu;

constexpr float kExtTmin = 0.001f;      // raygen.rgen.glsl:110
constexpr float kExtTmax = 10000.0f;
constexpr float kConnTmin = 0.0001f;    // lightSampling.glsl:112, next_event_estimation.glsl:3
constexpr int kCandidateCap = 1024;     // per-segment candidate bound for any-hit loops

// One atomic per warp for a per-lane count. All 32 lanes call it.
__device__ __forceinline__ void warp_add(uint32_t *counter, uint32_t v)
{
    const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31u) == 0 && sum)
        atomicAdd(counter, sum);
}

// Warp-aggregated queue append. Must be called by all 32 lanes of the warp
// at a convergence point (the kernels below keep their loop bounds
// warp-uniform); lanes with want == false get no slot.
__device__ __forceinline__ uint32_t warp_append_all(bool want, uint32_t *counter)
{
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, want);
    const int lane = threadIdx.x & 31;
    const int leader = mask ? __ffs(mask) - 1 : 0;
    uint32_t base = 0;
    if (want && lane == leader)
        base = atomicAdd(counter, (uint32_t)__popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    return base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

// K appends at once, in the same way: lane k makes the atomic of kind k, so a
// warp waits for one atomic's latency instead of K one after the other.
template <int K>
__device__ __forceinline__ void warp_append_many(const bool (&want)[K], uint32_t *const (&counter)[K],
                                                 uint32_t (&pos)[K])
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t mask[K], mine = 0, base = 0;
    uint32_t *to = nullptr;
#pragma unroll
    for (int k = 0; k < K; k++) {
        mask[k] = __ballot_sync(0xFFFFFFFFu, want[k]);
        if (lane == (uint32_t)k) {
            mine = mask[k];
            to = counter[k];
        }
    }
    if (mine)
        base = atomicAdd(to, (uint32_t)__popc(mine));
#pragma unroll
    for (int k = 0; k < K; k++)
        pos[k] = __shfl_sync(0xFFFFFFFFu, base, k) + (uint32_t)__popc(mask[k] & ((1u << lane) - 1u));
}

__device__ __forceinline__ float4 mat4_mul(const float4 *cols, float x, float y, float z, float w)
{
    return make_float4(cols[0].x * x + cols[1].x * y + cols[2].x * z + cols[3].x * w,
                       cols[0].y * x + cols[1].y * y + cols[2].y * z + cols[3].y * w,
                       cols[0].z * x + cols[1].z * y + cols[2].z * z + cols[3].z * w,
                       cols[0].w * x + cols[1].w * y + cols[2].w * z + cols[3].w * w);
}

// ---------------------------------------------------------------------------
// Hit reconstruction (shaders/pt/process_hit.glsl:1-17, construct_frame.glsl:1-15)

struct SurfaceHit {
    float3 wpos;
    float2 uv;
    Frame frame;
    bool flipped;
    uint32_t material;
    int32_t front_volume, back_volume;
};

__device__ __forceinline__ void fetch_triangle(const SceneView &s, const DevInstance &inst, uint32_t prim,
                                               ShadeVertex &a, ShadeVertex &b, ShadeVertex &c)
{
    const uint32_t *ix = s.indices + inst.index_offset + 3u * prim;
    uint32_t i0 = __ldg(ix), i1 = __ldg(ix + 1), i2 = __ldg(ix + 2);
    const ShadeVertex *v = s.verts + inst.vertex_offset;
    const float4 *p0 = reinterpret_cast<const float4 *>(v + i0);
    const float4 *p1 = reinterpret_cast<const float4 *>(v + i1);
    const float4 *p2 = reinterpret_cast<const float4 *>(v + i2);
    a.pos_u = __ldg(p0); a.nrm_v = __ldg(p0 + 1); a.tan_ = __ldg(p0 + 2);
    b.pos_u = __ldg(p1); b.nrm_v = __ldg(p1 + 1); b.tan_ = __ldg(p1 + 2);
    c.pos_u = __ldg(p2); c.nrm_v = __ldg(p2 + 1); c.tan_ = __ldg(p2 + 2);
}

__device__ __forceinline__ Affine34 rows_of(const float4 *r) { return Affine34{r[0], r[1], r[2]}; }

// Full hit record with the shading frame; `ray_dir` is gl_WorldRayDirectionEXT.
__device__ __forceinline__ SurfaceHit make_surface_hit(const SceneView &s, uint32_t inst_id, uint32_t prim, float hu,
                                                       float hv, const float3 &ray_dir)
{
    const DevInstance &inst = s.instances[inst_id];
    ShadeVertex a, b, c;
    fetch_triangle(s, inst, prim, a, b, c);
    const float bx = 1.0f - hu - hv, by = hu, bz = hv;
    SurfaceHit h;
    h.uv = make_float2(a.pos_u.w * bx + b.pos_u.w * by + c.pos_u.w * bz, a.nrm_v.w * bx + b.nrm_v.w * by + c.nrm_v.w * bz);
    float3 lp = f3(a.pos_u) * bx + f3(b.pos_u) * by + f3(c.pos_u) * bz;
    Affine34 o2w = rows_of(inst.o2w), w2o = rows_of(inst.w2o);
    h.wpos = xform_point(o2w, lp);
    float3 ln = f3(a.nrm_v) * bx + f3(b.nrm_v) * by + f3(c.nrm_v) * bz;
    float3 lt = f3(a.tan_) * bx + f3(b.tan_) * by + f3(c.tan_) * bz;
    h.frame.n = normalize3(xform_normal_transposed(w2o, ln));
    h.frame.t = normalize3(xform_normal_transposed(w2o, lt));
    h.frame.b = f3(0.0f, 0.0f, 1.0f); // overwritten by fix_frame in both branches
    h.flipped = fix_frame(h.frame, ray_dir);
    h.material = inst.material;
    h.front_volume = inst.front_volume;
    h.back_volume = inst.back_volume;
    return h;
}

__device__ __forceinline__ float3 material_emissive(const SceneView &s, const DevMaterial &m, float2 tuv)
{
    float4 te = tex2d(s, m.tex2[0], tuv.x, tuv.y);
    return (m.emissive.w * f3(m.emissive)) * f3(te);
}
__device__ __forceinline__ float material_alpha(const SceneView &s, const DevMaterial &m, float2 tuv)
{
    return m.albedo.w * tex2d(s, m.tex2[3], tuv.x, tuv.y).x;
}


// ---------------------------------------------------------------------------
// Light sampling (shaders/pt/lightSampling.glsl:1-106), without the shadow
// trace, which `connect` performs.

// ---- Sampler. RTGEMS (default): the xorshift stream of
// shaders/include/rng/rng_def.glsl:4-36, rand2D = two rand1D draws.
// PMJ (VVPT_RENDER_SAMPLER_PMJ): shaders/include/rng/rng_pmj.glsl:20-107,
// whose state is the pixel, the sample index and a dimension counter.
struct PathRng {
    uint32_t s;     // RTGEMS xorshift state, or the PMJ dimension
    uint32_t pix;   // PMJ: pixel x | y << 16
    uint32_t index; // PMJ: sample index within the pixel
};

// 64-bit finaliser, rng_pmj.glsl:28-35
__device__ __forceinline__ uint64_t pmj_mix_bits(uint64_t v)
{
    v ^= v >> 31;
    v *= 9202493588570546565ull;
    v ^= v >> 27;
    v *= 9357036318526133325ull;
    v ^= v >> 33;
    return v;
}

// Element i of a pseudo-random permutation of [0, l) keyed by p (cycle
// walking over the next power of two), rng_pmj.glsl:37-64. The walk ends
// within a few steps; the cap only guards the loop.
__device__ __forceinline__ uint32_t pmj_permutation_element(uint32_t i, uint32_t l, uint32_t p)
{
    uint32_t w = l - 1;
    w |= w >> 1;
    w |= w >> 2;
    w |= w >> 4;
    w |= w >> 8;
    w |= w >> 16;
    for (int it = 0; it < 1024; it++) {
        i ^= p;
        i *= 0xe170893du;
        i ^= p >> 16;
        i ^= (i & w) >> 4;
        i ^= p >> 8;
        i *= 0x0929eb3fu;
        i ^= p >> 23;
        i ^= (i & w) >> 1;
        i *= 1u | p >> 27;
        i *= 0x6935fa69u;
        i ^= (i & w) >> 11;
        i *= 0x74dcb303u;
        i ^= (i & w) >> 2;
        i *= 0x9e501cc3u;
        i ^= (i & w) >> 2;
        i *= 0xc860a3dfu;
        i &= w;
        i ^= i >> 5;
        if (i < l)
            break;
    }
    return (i + p) % l;
}

constexpr uint32_t kPmjSeed = 2873468793u;
constexpr float kOneMinusEpsilon = 0.999999f; // ONEMINUSEPSILON, shaders/include/constants.glsl:2

__device__ __forceinline__ uint32_t pmj_hash(const PathRng &r)
{
    const uint64_t px = r.pix & 0xFFFFu, py = r.pix >> 16;
    return (uint32_t)pmj_mix_bits((px << 48) ^ (py << 32) ^ ((uint64_t)r.s << 16) ^ (uint64_t)kPmjSeed);
}

__device__ __forceinline__ float rnd1(const RenderParams &p, PathRng &r)
{
    if (!p.sampler)
        return rand1(r.s);
    const uint32_t index = pmj_permutation_element(r.index, p.total_samples, pmj_hash(r));
    const uint32_t px = (r.pix & 0xFFFFu) % 128u, py = (r.pix >> 16) % 128u;
    const float delta = __ldg(p.blue_noise + ((size_t)(r.s % 48u) * 128u + px) * 128u + py);
    r.s++;
    return fminf(__fdiv_rn(__fadd_rn((float)index, delta), (float)p.total_samples), kOneMinusEpsilon);
}

__device__ __forceinline__ float2 rnd2(const RenderParams &p, PathRng &r)
{
    if (!p.sampler) {
        const float a = rand1(r.s);
        const float b = rand1(r.s);
        return make_float2(a, b);
    }
    uint32_t index = r.index;
    const uint32_t inst = r.s / 2u;
    if (inst >= 16u)
        index = pmj_permutation_element(r.index, p.total_samples, pmj_hash(r));
    const float2 u = __ldg(reinterpret_cast<const float2 *>(p.pmj) + (size_t)(inst % 16u) * 16384u + index % 16384u);
    r.s += 2u;
    return make_float2(fminf(u.x, kOneMinusEpsilon), fminf(u.y, kOneMinusEpsilon));
}

// Two neighbouring members of a slot's state in one 32-byte access.
__device__ __forceinline__ void load_pair(const float4 &at, float4 &a, float4 &b)
{
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(&at));
}
__device__ __forceinline__ void store_pair(float4 &at, const float4 &a, const float4 &b)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(&at), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

// The path's sampler state as the shade kernels use it.
__device__ __forceinline__ PathRng load_rng(const RenderParams &p, const PathState &ps, uint32_t slot, uint32_t state)
{
    PathRng r;
    r.s = state;
    r.pix = 0;
    r.index = 0;
    if (p.sampler) {
        const uint32_t npix = p.width * p.height, item = __float_as_uint(ps[slot].cum_rad.w);
        const uint32_t batch = item / npix, pix = item - batch * npix;
        r.pix = (pix % p.width) | ((pix / p.width) << 16);
        r.index = batch * p.batch_size + __float_as_uint(ps[slot].cum_alb.w);
    }
    return r;
}

struct LightSample {
    float3 dir;
    float3 radiance;
    float pdf;
    float tmax;
    bool delta;
};

// With env_light set, the environment is light number num_lights of the
// uniform pick (importance sampled by sample_env); `allow_env` = false makes
// that pick contribute nothing (the last event of a path, whose environment
// contribution the reference's estimator never adds either).
// Out of line with VVPT_SHADE_OUTLINE = 1 (a build option, measured, not
// kept): the shading kernel samples a light at a medium scatter point and at
// a surface, and one copy instead of two shortens its instruction stream,
// but the call's register saves cost more (1920 x 1080 x 64 medium scene:
// 158.0 against 160.0 M paths/s).
#ifndef VVPT_SHADE_OUTLINE
#define VVPT_SHADE_OUTLINE 0
#endif
#if VVPT_SHADE_OUTLINE
#define VVPT_SHADE_FN __noinline__
#else
#define VVPT_SHADE_FN __forceinline__
#endif
__device__ VVPT_SHADE_FN LightSample sample_light(const SceneView &s, const RenderParams &p, const float3 origin,
                                                  PathRng &rng, bool allow_env)
{
    LightSample ls;
    ls.delta = true;
    ls.radiance = f3(0.0f);
    ls.pdf = 1.0f;
    ls.dir = f3(0.0f);
    ls.tmax = 10000.0f;
    const uint32_t total = p.num_lights + p.env_light;
    if (total == 0)
        return ls;
    float pdf = 1.0f / (float)total;
    uint32_t li = (uint32_t)(rnd1(p, rng) * (float)total);
    if (li >= total)
        li = total - 1;
    if (li == p.num_lights) {
        ls.delta = false;
        if (!allow_env)
            return ls;
        const float2 uv = rnd2(p, rng);
        const float u_row = uv.x, u_col = uv.y;
        float epdf;
        ls.dir = sample_env(s, u_row, u_col, epdf);
        ls.tmax = p.zfar;
        if (epdf > 0.0f) {
            ls.radiance = env_lookup(s, ls.dir) * ((int)p.env_type == 1 ? p.env_intensity : 1.0f);
            ls.pdf = pdf * epdf;
        }
        return ls;
    }
    const DevLightInstance &L = s.lights[li];
    const uint32_t type = L.info[3];
    if (type == 0) {
        float3 lp = f3(L.position);
        float3 dir = lp - origin;
        float tmax = length3(dir);
        ls.tmax = tmax;
        ls.dir = dir / tmax;
        float dist = length3(origin - lp);
        ls.radiance = f3(L.color) * (1.0f / (dist * dist)) * L.color.w;
        ls.pdf = pdf * 1.0f;
        ls.delta = true;
    } else if (type == 1) {
        ls.dir = -f3(L.position);
        ls.tmax = p.zfar;
        ls.radiance = f3(L.color) * L.color.w;
        ls.pdf = pdf * 1.0f;
        ls.delta = true;
    } else if (type == 2) {
        const uint32_t mesh_inst = L.info[1];
        const DevInstance &inst = s.instances[mesh_inst];
        const DevMaterial &m = s.materials[inst.material];
        uint32_t tri = (uint32_t)(rnd1(p, rng) * (float)inst.num_triangles);
        if (tri >= inst.num_triangles)
            tri = inst.num_triangles - 1;
        float tri_pdf = 1.0f / (float)inst.num_triangles;
        const float2 uu = rnd2(p, rng);
        float2 bc = uniform_sample_triangle(uu.x, uu.y);
        float b0 = bc.x, b1 = bc.y, b2 = 1.0f - bc.x - bc.y;
        ShadeVertex a, b, c;
        fetch_triangle(s, inst, tri, a, b, c);
        Affine34 M{L.position, L.position1, L.position2};
        float3 p0 = xform_point(M, f3(a.pos_u)), p1 = xform_point(M, f3(b.pos_u)), p2 = xform_point(M, f3(c.pos_u));
        float area = 0.5f * length3(cross3(p1 - p0, p2 - p0));
        float point_pdf = 1.0f / area;
        float3 sp = f3(a.pos_u) * b0 + f3(b.pos_u) * b1 + f3(c.pos_u) * b2;
        float3 sn = f3(a.nrm_v) * b0 + f3(b.nrm_v) * b1 + f3(c.nrm_v) * b2;
        float2 suv = make_float2(a.pos_u.w * b0 + b.pos_u.w * b1 + c.pos_u.w * b2,
                                 a.nrm_v.w * b0 + b.nrm_v.w * b1 + c.nrm_v.w * b2);
        sp = xform_point(M, sp);
        Affine34 N{L.nrm0, L.nrm1, L.nrm2};
        sn = xform_vector(N, sn);
        float3 dir = sp - origin;
        float tmax = length3(dir);
        ls.tmax = tmax;
        ls.dir = dir / tmax;
        float dp = dot3(-ls.dir, sn);
        if (dp > 0.0f) {
            float2 tuv = make_float2(suv.x * m.uv_tiling.x, suv.y * m.uv_tiling.y);
            ls.radiance = material_emissive(s, m, tuv);
            float dist = length3(origin - sp);
            ls.pdf = pdf * tri_pdf * point_pdf * (dist * dist) / dp;
        } else {
            ls.radiance = f3(0.0f);
            ls.pdf = 0.0f;
        }
        ls.delta = false;
    }
    return ls;
}

// ---------------------------------------------------------------------------
// Homogeneous medium free flight (shaders/pt/process_volume_hit.glsl:1-40)

struct Medium {
    float3 sigma_s, sigma_t;
    float g;
};
__device__ __forceinline__ Medium load_medium(const SceneView &s, uint32_t vol)
{
    const DevMaterial &m = s.materials[vol];
    Medium md;
    float3 sa = f3(m.albedo);
    md.sigma_s = fmax3(f3(m.mrao), kEps);
    md.sigma_t = sa + md.sigma_s;
    md.g = fmaxf(fminf(m.emissive.x, 0.99f), -0.99f);
    return md;
}
// process_volume_transmittance.glsl:1-9
__device__ __forceinline__ float3 medium_transmittance(const SceneView &s, uint32_t vol, float vtstart, float vtend)
{
    const DevMaterial &m = s.materials[vol];
    float3 ss = fmax3(f3(m.mrao), kEps);
    float3 st = f3(m.albedo) + ss;
    float dist = fmaxf(vtend - vtstart, kEps);
    return f3(expf(-st.x * dist), expf(-st.y * dist), expf(-st.z * dist));
}

// ---------------------------------------------------------------------------
// Kernels

// The job of a path. A render has one, which its kernels get as a parameter
// (kOne): its fields are then operands in constant memory instead of loads
// through the table, of which every traversal step needs one before its node
// and a shading event dozens (1080p x 32 medium scene 162.1 to 156.2 ms, 64-sample
// Cornell box 8.44 to 8.07, 256 x 256 preview 2.37 to 2.25).
template <bool kOne>
__device__ __forceinline__ const JobView &job_view(const JobTable &jt, const JobView &one, uint32_t job)
{
    return kOne ? one : jt.jobs[job];
}

__global__ void k_init_slots(Queues q, PathState ps, JobTable jt, uint32_t slots)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += gridDim.x * blockDim.x) {
        q.regen[0][i] = i;
        ps[i].flags = 0u;
        ps[i].cum_rad.w = __uint_as_float(0xFFFFFFFFu);
        ps[i].job = 0u;
    }
    if (blockIdx.x == 0)
        vvpt_srgb_lut[threadIdx.x & 255u] = srgb_to_linear((float)(threadIdx.x & 255u) / 255.0f);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int c = 0; c < C_COUNT; c++)
            q.counters[c] = 0u;
        q.counters[C_REGEN0] = slots;
        *jt.next_item = 0ull;
        *jt.idle_count = 0u;
    }
}

// New work for idle slots (see launch_admit). One block: the counters it
// resets are read by all of its threads first.
__global__ void k_admit(Queues q, JobTable jt, unsigned long long total_items, uint32_t num_ranges)
{
    const uint32_t n = *jt.idle_count;
    const uint32_t base = q.counters[C_REGEN0];
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
        q.regen[0][base + i] = jt.idle[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        // hand-out attempts past the old end claimed nothing
        const unsigned long long old_total = *jt.total_items;
        if (*jt.next_item > old_total)
            *jt.next_item = old_total;
        *jt.total_items = total_items;
        *jt.num_ranges = num_ranges;
        q.counters[C_REGEN0] = base + n;
        *jt.idle_count = 0u;
    }
}

// Hand-out range holding global work item g (the last range beginning at or
// before g).
__device__ __forceinline__ uint32_t find_range(const JobTable &jt, uint32_t num_ranges, unsigned long long g)
{
    uint32_t lo = 0, hi = num_ranges;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jt.range_begin[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Finalizes finished samples, hands out work items, and generates camera
// rays (raygen.rgen.glsl:24-99, 126-129).
// Bound by memory latency: a slot's state is loaded at once, before anything
// depends on it, the counters take two rounds of atomics per warp, and what a
// sample leaves as it is is not written back (246,000 paths: 108 -> 98 us; the
// reset of the counters rides along instead of being a launch of its own).
template <bool kOne>
__global__ void __launch_bounds__(256)
    k_regen(JobTable jt, PathState ps, Queues q, int pp, const __grid_constant__ JobView one)
{
    const uint32_t n = q.counters[C_REGEN0 + pp];
    const uint32_t *queue = q.regen[pp];
    const unsigned long long total_items = *jt.total_items;
    const uint32_t num_ranges = *jt.num_ranges;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // queues of the previous iteration, consumed by now, that this
        // iteration's later kernels fill
        q.counters[C_SHADE_L] = 0u;
        q.counters[C_SHADE_P] = 0u;
        q.counters[C_SHADE_M] = 0u;
        q.counters[C_WALK] = 0u;
        q.counters[C_FETCH] = 0u;
        q.counters[C_EXT0 + (1 - pp)] = 0u;
    }
    // The loop bound is warp-uniform: the counters below take one atomic per
    // warp (one per job for finished items) instead of one per slot, as the
    // slots of a launch all update the same few addresses.
    // Those that nothing in the launch reads are added up over the loop and take
    // one per warp and launch (the 1080p x 32 medium scene: 16.6 to 14.5 ms of
    // regeneration).
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t paths = 0, active = 0;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < n;
        uint32_t slot = 0, flags = 0, sample = 0, item = 0, job = 0, rng_state = 0;
        float3 cr = f3(0.0f), ca = f3(0.0f), cn = f3(0.0f), rad = f3(0.0f), alb = f3(0.0f), nrm = f3(0.0f);
        bool path_done = false, item_done = false;
        if (valid) {
            slot = queue[i];
            const uint4 meta = ps[slot].meta;
            float4 a, b, c, d, e, f;
            load_pair(ps[slot].cum_rad, a, b);
            load_pair(ps[slot].beta, c, d);
            load_pair(ps[slot].alb, e, f);
            cn = f3(ps[slot].cum_nrm);
            flags = meta.x;
            job = meta.z;
            cr = f3(a);
            item = __float_as_uint(a.w);
            ca = f3(b);
            sample = __float_as_uint(b.w);
            rng_state = __float_as_uint(c.w);
            rad = f3(d);
            alb = f3(e);
            nrm = f3(f);
            if (flags & F_DONE) {
                const float total = (float)job_view<kOne>(jt, one, job).params.total_samples;
                float3 r = rad;
                if (flags & F_NEE) // the emitter ray's contribution, after the shadow ray's
                    r = r + f3(ps[slot].nee_c);
                cr += r / total;
                ca += alb / total;
                cn += nrm / total;
                sample++;
                path_done = true;
            }
            if ((flags & F_ITEM) && sample >= job_view<kOne>(jt, one, job).params.batch_size) {
                // the item's batch sums; the host and k_reduce read them after
                // this launch, in stream order
                const BatchResults br = job_view<kOne>(jt, one, job).results;
                br.rad[item] = f4(cr, 1.0f);
                br.alb[item] = f4(ca, 1.0f);
                br.nrm[item] = f4(cn, 1.0f);
                flags &= ~F_ITEM;
                item_done = true;
            }
        }
        paths += path_done ? 1u : 0u;
        const uint32_t fin = __ballot_sync(0xFFFFFFFFu, item_done);
        if (item_done) {
            const uint32_t same = __match_any_sync(fin, job);
            if (lane == (uint32_t)(__ffs(same) - 1))
                atomicAdd(&jt.item_done[job], (uint32_t)__popc(same));
        }
        // next work items, in lane order, for the slots without one
        const bool need = valid && !(flags & F_ITEM);
        const uint32_t need_mask = __ballot_sync(0xFFFFFFFFu, need);
        unsigned long long g0 = 0;
        if (lane == 0 && need_mask)
            g0 = atomicAdd(jt.next_item, (unsigned long long)__popc(need_mask));
        g0 = __shfl_sync(0xFFFFFFFFu, g0, 0);
        const unsigned long long g = g0 + (unsigned long long)__popc(need_mask & ((1u << lane) - 1u));
        const bool got = need && g < total_items;
        const bool idle = need && !got;
        active += (got ? 1u : 0u) - (item_done ? 1u : 0u); // mod 2^32
        const bool emit = valid && !idle;
        uint32_t pos[2];
        warp_append_many<2>({idle, emit}, {jt.idle_count, &q.counters[C_EXT0 + pp]}, pos);
        if (idle) {
            ps[slot].flags = 0u;
            ps[slot].cum_rad.w = __uint_as_float(0xFFFFFFFFu);
            jt.idle[pos[0]] = slot;
        } else if (valid) {
            // camera ray of a slot that holds a work item (a new item's sums
            // and RNG state start from zero)
            q.ext[pp][pos[1]] = slot;
            if (got) {
                const uint32_t r = find_range(jt, num_ranges, g);
                item = (uint32_t)(g - jt.range_begin[r]);
                job = jt.range_job[r];
                sample = 0;
                cr = ca = cn = f3(0.0f);
            }
            const RenderParams &p = job_view<kOne>(jt, one, job).params;
            const uint32_t npix = p.width * p.height;
            const uint32_t batch = item / npix;
            const uint32_t pix = item - batch * npix;
            const uint32_t px = pix % p.width, py = pix / p.width;
            PathRng rng;
            rng.s = got ? init_rng(px, py, p.width, batch) : rng_state;
            rng.pix = px | (py << 16);
            rng.index = batch * p.batch_size + sample;
            if (p.sampler)
                rng.s = py * p.width + py; // dimension start of every sample, raygen.rgen.glsl:57-60
            // camera ray, raygen.rgen.glsl:63-91
            const float2 oxy = rnd2(p, rng);
            const float ox = oxy.x, oy = oxy.y;
            float uvx = ((float)px + ox) / (float)p.width;
            float uvy = ((float)py + oy) / (float)p.height;
            float dx = uvx * 2.0f - 1.0f, dy = uvy * 2.0f - 1.0f;
            float4 target = mat4_mul(p.proj_inv, dx, dy, 1.0f, 1.0f);
            float3 dcam = normalize3(f3(target.x, target.y, target.z));
            float3 ocam = f3(0.0f);
            if (p.lens_radius > 0.0f) {
                const float2 lxy = rnd2(p, rng);
                const float lx = lxy.x, ly = lxy.y;
                float2 disk = concentric_sample_disk(lx, ly);
                float2 lens = make_float2(p.lens_radius * disk.x, p.lens_radius * disk.y);
                float ft = p.focal_distance / (-dcam.z);
                float3 focus = dcam * ft;
                ocam = f3(lens.x, lens.y, 0.0f);
                dcam = normalize3(focus - ocam);
            }
            float4 wo = mat4_mul(p.view_inv, ocam.x, ocam.y, ocam.z, 1.0f);
            float4 wd = mat4_mul(p.view_inv, dcam.x, dcam.y, dcam.z, 0.0f);
            uint32_t nf = F_ITEM;
            if (p.cam_volume != -1)
                nf |= F_INSIDE;
            ps[slot].meta = make_uint4(nf, (uint32_t)p.cam_volume, job, kNoHit);
            store_pair(ps[slot].o, make_float4(wo.x, wo.y, wo.z, 0.0f), make_float4(wd.x, wd.y, wd.z, 0.0f));
            store_pair(ps[slot].beta, make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(rng.s)),
                       make_float4(0.0f, 0.0f, 0.0f, 0.0f));
            store_pair(ps[slot].cum_rad, f4(cr, __uint_as_float(item)), f4(ca, __uint_as_float(sample)));
            ps[slot].cum_nrm = f4(cn, 0.0f);
            if (got) // first-hit albedo and normal carry over from sample to sample of an item and start from zero
                store_pair(ps[slot].alb, make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        }
    }
    warp_add(&q.counters[C_PATHS], paths);
    warp_add(&q.counters[C_ACTIVE], active);
}

// Minimum resident blocks of 256 threads per SM requested for the traversal
// kernels, which caps their registers (k_trace 5: 48 registers; k_walk 4: 64).
// What k_trace waits for most is its loads, and the fifth block, which the ray
// state in shared memory makes room for without spills in the loop, covers
// more of that: 161 -> 149 ms on the 1080p medium scene, 41.0 -> 38.9 ms on
// the sky scene.
#ifndef VVPT_TRACE_MIN_BLOCKS
#define VVPT_TRACE_MIN_BLOCKS 5
#endif
#ifndef VVPT_WALK_MIN_BLOCKS
#define VVPT_WALK_MIN_BLOCKS 4
#endif
#ifndef VVPT_SHADE_MIN_BLOCKS
#define VVPT_SHADE_MIN_BLOCKS 2
#endif
// the Lambert and miss shading kernels
#ifndef VVPT_SHADE_LM_MIN_BLOCKS
#define VVPT_SHADE_LM_MIN_BLOCKS 2
#endif
__device__ __forceinline__ uint32_t first_ray() { return blockIdx.x * blockDim.x; }
__device__ __forceinline__ uint32_t my_ray() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t ray_stride() { return gridDim.x * blockDim.x; }

// Shade bin of a closest hit (0 Lambert, 1 PBR, 2 miss; | 4: the fused
// emitter ray takes the full candidate walk).
__device__ __forceinline__ uint32_t extend_key(const SceneView &s, const Hit &h, bool fused, uint32_t key)
{
    if (h.inst == kNoHit)
        return key | 2u;
    const DevMaterial &m = s.materials[s.instances[h.inst].material];
    key |= (uint32_t)m.uv_tiling.z == 2u ? 0u : 1u;
    // a transparent first candidate also needs the walk
    if (fused && h.t <= kExtTmax && m.mrao.w >= 0.99f)
        key |= 4u;
    return key;
}

// Lane refill: a warp traces its rays step by step (trace_step). A lane is
// free, tracing, or done (its traversal ended, its result not yet used).
// When no more than VVPT_REFILL_BELOW of the warp's lanes are tracing, the
// done lanes finish their rays together and the free lanes take the next
// rays of the queue (one atomic per warp). Rays of very different lengths
// then share a warp's steps instead of the warp running until its longest
// ray ends, and the code between traversals runs for many lanes at once.
// Per-lane values that only that code reads stay in shared memory (one entry
// per thread), so the traversal state keeps the registers.
#ifndef VVPT_REFILL_BELOW
#define VVPT_REFILL_BELOW 20
#endif
constexpr uint32_t kLaneFree = 0, kLaneTracing = 1, kLaneDone = 2;
// Step turns: triangle tests and transitions between the levels wait until
// enough lanes share them. Triangle tests when at least VVPT_TRI_TURN_PCT % of
// the tracing lanes have one pending, else transitions when at least
// VVPT_LEVEL_TURN_PCT % have (or no lane has a node to visit). Entering an
// instance is a hundred instructions that nearly every warp step executed for
// one or two lanes: in turns of their own, trace launches of the 1080p medium
// scene (32 spp) 167 -> 159 ms, of the sky scene 44.1 -> 40.7 ms (thresholds of
// 10, 25 and 40 %: 163, 159, 159 ms).
// Within a turn a lane takes up to kTriSteps triangles and then up to
// kNodeSteps nodes, without another vote: the two ballots and the comparisons
// of a vote cost about half as much as a node visit, and most lanes that visit
// a node visit another. One step a turn, one kind of step a turn: 185 ms on the
// 1080p x 32 medium scene, 50.8 ms on the sky scene, 9.6 ms on the 64-sample
// Cornell box; these: 170, 48.8 and 9.0 ms (two nodes 178, 49.4 and 9.4; eight
// 178, 49.1 and 9.2; three triangles 175, 48.9 and 9.1).
constexpr int kTriSteps = 2, kNodeSteps = 4;
#ifndef VVPT_TRI_TURN_PCT
#define VVPT_TRI_TURN_PCT 33
#endif
#ifndef VVPT_LEVEL_TURN_PCT
#define VVPT_LEVEL_TURN_PCT 33
#endif
// (a turn always has a lane that steps, so the loop ends)
static_assert(VVPT_TRI_TURN_PCT > 0 && VVPT_TRI_TURN_PCT <= 100, "share of the tracing lanes, in percent");

// Hands the next queue entries to the free lanes of the warp: returns the
// entry index of this lane (meaningful when `mine`), and clears `open` when
// the queue has no entries left after these. Warp-uniform call.
__device__ __forceinline__ uint32_t refill_take(bool free, uint32_t *counter, uint32_t n, bool &open, bool &mine)
{
    const uint32_t want = __ballot_sync(0xFFFFFFFFu, free);
    const uint32_t cnt = (uint32_t)__popc(want);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t base = 0;
    if (lane == 0 && cnt)
        base = atomicAdd(counter, cnt);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (cnt)
        open = base + cnt < n;
    const uint32_t idx = base + (uint32_t)__popc(want & ((1u << lane) - 1u));
    mine = free && idx < n;
    return idx;
}

// One turn of the refill loops over their `all` tracing lanes: triangle tests or
// transitions where enough lanes wait for them, then node visits (every kind
// gets its turn, since the lanes that step move on to another kind, finish, or
// leave the tracing set). True when this lane's traversal ended.
__device__ __forceinline__ bool trace_turn(TraceState &st, const TraceCold &ray, TraceStack &stack, const SceneView &s,
                                           bool tracing, int all, uint32_t &err)
{
    const int kind = tracing ? trace_kind(st) : -1;
    const int ntri = 100 * __popc(__ballot_sync(0xFFFFFFFFu, kind == kStepTriangle));
    const int nlev = 100 * __popc(__ballot_sync(0xFFFFFFFFu, kind == kStepLevel));
    if (ntri >= VVPT_TRI_TURN_PCT * all) {
#pragma unroll
        for (int r = 0; r < kTriSteps; r++)
            if (tracing && trace_kind(st) == kStepTriangle)
                trace_step_triangle(st, ray, stack, s, no_hit());
    } else if (nlev && (nlev >= VVPT_LEVEL_TURN_PCT * all || nlev + ntri == 100 * all)) {
        if (kind == kStepLevel)
            trace_step_level(st, ray, stack, s, err);
    }
#pragma unroll
    for (int r = 0; r < kNodeSteps; r++)
        if (tracing && trace_kind(st) == kStepNode)
            trace_step_node(st, stack, s, err);
    return tracing && st.cur == kRefDone;
}

// A shadow ray whose nearest candidate is known: opaque, the light is hidden;
// none, the light is seen through the medium at the event (the miss shader of
// raySecondary.rmiss.glsl:17-44); transparent, the candidates have to be
// walked (k_walk), which returns true.
__device__ __forceinline__ bool shadow_finish(const JobView &J, const PathState &ps, uint32_t slot, const Hit &h)
{
    const SceneView &s = J.scene;
    if (h.inst != kNoHit) {
        if (!(s.materials[s.instances[h.inst].material].mrao.w >= 0.99f))
            return false;
        ps[slot].flags |= F_SHADOW_WALK;
        return true;
    }
    float3 T = f3(1.0f);
    if (ps[slot].flags & F_INSIDE) {
        const uint32_t vol = ps[slot].vol;
        if (vol < s.num_materials) {
            T *= medium_transmittance(s, vol, kConnTmin, fminf(J.params.zfar_trunc, h.t));
            if (!(max3f(T) > kEps))
                T = f3(0.0f);
        }
    }
    if (!is_black(T))
        ps[slot].rad = f4(f3(ps[slot].rad) + f3(ps[slot].sh_c) * T, 0.0f);
    return false;
}

// Closest hits: the extension rays of this iteration, then the shadow rays of
// the events shaded in the previous one and the emitter rays of the paths that
// ended there, from one hand-out sequence, so that all share the lane refill
// and a launch has one tail of long rays instead of three. Issue-bound under
// divergence, then bound by the latency of dependent node fetches. Measured
// against a shadow launch of its own after k_shade (one ray per lane to its
// end, walks and emitter rays inline): 1920 x 1080 x 32 medium scene, 143 ms
// of extension + 135 ms of shadow launches -> 211 ms; 4096 shadow rays under
// the open sky (512 instances) took 215 us a launch, nearly all of it the
// tail, and now disappear behind the extension rays: 106 -> 92 ms.
constexpr uint32_t kColdFused = 1u, kColdShadow = 2u, kColdEmitter = 4u; // cold[].z; shade-bin bits above them
template <bool kOne>
__global__ void __launch_bounds__(256, VVPT_TRACE_MIN_BLOCKS)
    k_trace(JobTable jt, PathState ps, Queues q, int pp, const __grid_constant__ JobView one)
{
    const uint32_t ne = q.counters[C_EXT0 + pp], ns = q.counters[C_CONN];
    const uint32_t n = ne + ns + q.counters[C_NEEQ];
    if (n == 0)
        return;
    uint32_t err = 0;
    auto entry = [&](uint32_t i) {
        return i < ne ? q.ext[pp][i] : (i < ne + ns ? q.conn[i - ne] : q.nee[i - ne - ns]);
    };
    tlas_cache_fill(job_view<kOne>(jt, one, ps[entry(min(first_ray(), n - 1u))].job).scene);
    // per lane: queue index, slot, kind of ray and shade-bin bits, job; the ray
    __shared__ uint4 cold[256];
    __shared__ float4 cold_o[256], cold_d[256], cold_best[256];
    __shared__ uint2 cold_ids[256];
    const TraceCold ray{cold_o[threadIdx.x], cold_d[threadIdx.x], cold_best[threadIdx.x], cold_ids[threadIdx.x]};
    TraceState st;
    TraceStack stack;
    uint32_t state = kLaneFree, job = 0;
    bool open = true; // warp-uniform: the queue may still hold rays
    // fewer rays than the grid has lanes: every warp takes its share, on its
    // first lanes, instead of some warps taking 32 and the rest none (256 x 256
    // previews, about 100,000 rays a launch: 49 -> 41 us a launch)
    const uint32_t warps = gridDim.x * blockDim.x / 32u;
    const uint32_t lanes = min(n / warps + 1u, 32u);
    const bool takes = (threadIdx.x & 31u) < lanes;
    for (;;) {
        uint32_t tr = __ballot_sync(0xFFFFFFFFu, state == kLaneTracing);
        if (__popc(tr) <= (open ? (int)(lanes * VVPT_REFILL_BELOW / 32u) : 0)) {
            uint32_t walk_slot = 0;
            bool walk = false;
            if (state == kLaneDone) {
                const uint4 c = cold[threadIdx.x];
                const Hit h = trace_best(ray);
                const uint32_t key = c.z >> 3;
                if (c.z & kColdShadow) {
                    walk = shadow_finish(job_view<kOne>(jt, one, job), ps, c.y, h);
                    walk_slot = c.y;
                    state = kLaneFree;
                } else if ((c.z & kColdFused) && key == 0 && h.inst != kNoHit && h.t < kExtTmin) {
                    // the emitter ray's first candidate lies below the
                    // extension ray's tmin: the emitter ray takes the full
                    // candidate walk, and this lane goes on with the
                    // extension ray from its tmin
                    cold[threadIdx.x].z = kColdFused | (4u << 3);
                    const float3 o = f3(ray.o_slack), d = f3(ray.d_tmin);
                    trace_begin(st, ray, job_view<kOne>(jt, one, job).scene, o, d, kExtTmin, kExtTmax, no_hit());
                    state = kLaneTracing;
                } else {
                    ps[c.y].hit = make_float4(h.t, h.u, h.v, __uint_as_float(h.prim));
                    ps[c.y].hit_inst = h.inst;
                    if (!(c.z & kColdEmitter))
                        q.ext_key[c.x] = extend_key(job_view<kOne>(jt, one, job).scene, h, (c.z & kColdFused) != 0, key);
                    state = kLaneFree;
                }
            }
            if (__any_sync(0xFFFFFFFFu, walk)) {
                const uint32_t pos = warp_append_all(walk, &q.counters[C_WALK]);
                if (walk)
                    q.walk[pos] = walk_slot;
            }
            if (open) {
                bool mine;
                const uint32_t i = refill_take(takes && state == kLaneFree, &q.counters[C_FETCH], n, open, mine);
                if (mine) {
                    const bool ext = i < ne, shadow = !ext && i < ne + ns;
                    const uint32_t slot = entry(i);
                    const uint4 meta = ps[slot].meta;
                    const uint32_t flags = shadow ? 0u : meta.x;
                    job = meta.z;
                    float4 o, d;
                    load_pair(ps[slot].o, o, d);
                    if (shadow)
                        d = ps[slot].sh_dir;
                    // with an emitter ray riding on the extension ray, start at its tmin
                    const bool fused = ext && (flags & F_NEE_FUSED) != 0;
                    cold[threadIdx.x] =
                        make_uint4(i, slot, shadow ? kColdShadow : (!ext ? kColdEmitter : (fused ? kColdFused : 0u)), 0u);
                    const float tmax = ext ? kExtTmax : (shadow ? d.w - kConnTmin : job_view<kOne>(jt, one, job).params.zfar);
                    // the emitter ray of a path that goes on (zfar beyond the
                    // extension rays' range) takes the walk as a whole: the
                    // path's hit record belongs to its extension ray
                    if (ext || shadow || (flags & F_DONE)) {
                        trace_begin(st, ray, job_view<kOne>(jt, one, job).scene, f3(o), f3(d),
                                    ext && !fused ? kExtTmin : kConnTmin, tmax, no_hit());
                        state = kLaneTracing;
                    }
                }
            }
            tr = __ballot_sync(0xFFFFFFFFu, state == kLaneTracing);
            if (tr == 0) {
                if (!open)
                    break;
                continue;
            }
        }
        if (trace_turn(st, ray, stack, job_view<kOne>(jt, one, job).scene, state == kLaneTracing, __popc(tr), err))
            state = kLaneDone;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&q.counters[C_SEGMENTS], ne);
        atomicAdd(&q.counters[C_SHADOW], ns);
    }
    if (err)
        atomicOr(&q.counters[C_ERR], err);
}

// Compacts the extension queue into the material-sorted shade queues and the
// emitter-walk queue. Its work is a few bytes per entry; what it waits for is
// its atomics, so a block takes four entries per thread and makes one atomic
// per queue for all of them (875,000 entries, one atomic per warp and queue:
// 47 us, per block of 1024: 14 us).
__global__ void __launch_bounds__(256) k_partition(PathState ps, Queues q, int pp)
{
    const uint32_t n = q.counters[C_EXT0 + pp];
    const uint32_t *queue = q.ext[pp];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // queues that are consumed by now and filled again by this
        // iteration's k_shade; the emitter rays' entries stay for k_walk
        q.counters[C_CONN] = 0u;
        q.counters[C_REGEN0 + pp] = 0u;
        q.counters[C_NEE_RUN] = q.counters[C_NEEQ];
        q.counters[C_NEEQ] = 0u;
    }
    constexpr int kPer = 4, kBins = 4; // Lambert, PBR, miss, walk
    __shared__ uint32_t at[8][kBins];  // per warp: entries, then its first position
    uint32_t *const counters[kBins] = {&q.counters[C_SHADE_L], &q.counters[C_SHADE_P], &q.counters[C_SHADE_M],
                                       &q.counters[C_WALK]};
    uint32_t *const to[kBins] = {q.shade_l, q.shade_p, q.shade_m, q.walk};
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    const uint32_t per_block = kPer * blockDim.x;
    for (uint32_t base = blockIdx.x * per_block; base < n; base += gridDim.x * per_block) {
        uint32_t slot[kPer], key[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const uint32_t i = base + (warp * kPer + k) * 32u + lane;
            slot[k] = i < n ? queue[i] : 0u;
            key[k] = i < n ? q.ext_key[i] : 3u;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++)
            if (key[k] & 4u) {
                // one walk entry per path: a shadow walk's entry serves both
                const uint32_t flags = ps[slot[k]].flags;
                ps[slot[k]].flags = flags | F_NEE_FULL;
                if (flags & F_SHADOW_WALK)
                    key[k] &= 3u;
            }
        uint32_t count = 0; // lane b: the warp's entries of bin b
#pragma unroll
        for (int k = 0; k < kPer; k++)
#pragma unroll
            for (int b = 0; b < kBins; b++) {
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, b < 3 ? (key[k] & 3u) == (uint32_t)b : (key[k] & 4u) != 0);
                if (lane == (uint32_t)b)
                    count += (uint32_t)__popc(m);
            }
        if (lane < kBins)
            at[warp][lane] = count;
        __syncthreads();
        if (threadIdx.x < kBins) {
            uint32_t sum = 0;
            for (uint32_t w = 0; w < blockDim.x / 32u; w++)
                sum += at[w][lane];
            uint32_t pos = sum ? atomicAdd(counters[lane], sum) : 0u;
            for (uint32_t w = 0; w < blockDim.x / 32u; w++) {
                const uint32_t c = at[w][lane];
                at[w][lane] = pos;
                pos += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int b = 0; b < kBins; b++) {
            uint32_t pos = at[warp][b];
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const bool in = b < 3 ? (key[k] & 3u) == (uint32_t)b : (key[k] & 4u) != 0;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, in);
                if (in)
                    to[b][pos + (uint32_t)__popc(m & below)] = slot[k];
                pos += (uint32_t)__popc(m);
            }
        }
        __syncthreads(); // `at` is filled again
    }
}

// Volume free flight on the current segment; returns true when the path
// scattered in the medium (sampledMedium) and writes the scatter point.
__device__ __forceinline__ bool medium_event(const SceneView &s, const RenderParams &p, uint32_t vol, float vtstart,
                                             float vtend, const float3 &origin, const float3 &raydir, float3 &beta,
                                             PathRng &rng, float3 &scatter_pos, float &g)
{
    Medium md = load_medium(s, vol);
    g = md.g;
    float3 dirn = normalize3(raydir);
    float dist_in = fmaxf(vtend - vtstart, kEps);
    uint32_t channel = min((uint32_t)(rnd1(p, rng) * 3.0f), 2u);
    float u = rnd1(p, rng);
    float hit_dist = -logf(1.0f - u) / comp(md.sigma_t, channel);
    bool sampled = hit_dist < dist_in;
    float td = fminf(hit_dist, dist_in);
    float3 tr = f3(expf(-md.sigma_t.x * td), expf(-md.sigma_t.y * td), expf(-md.sigma_t.z * td));
    float3 density = sampled ? md.sigma_t * tr : tr;
    float pdf = 0.0f;
    pdf += density.x;
    pdf += density.y;
    pdf += density.z;
    pdf *= 0.3333333f;
    if (pdf == 0.0f)
        pdf = 1.0f;
    float3 F = sampled ? (tr * md.sigma_s / pdf) : (tr / pdf);
    beta *= F;
    if (sampled)
        scatter_pos = origin + (vtstart + hit_dist) * dirn;
    return sampled;
}

__device__ __noinline__ float3 fused_nee(const SceneView &s, const RenderParams &p, bool full, bool is_hit,
                                         uint32_t inst_id, float4 hv, float3 o, float3 dir, bool inside, uint32_t vol,
                                         float4 nb, uint32_t &err, uint32_t &walks);

// One shading event per queued path: the body of rayPrimary*.rchit.glsl:45-175
// (hits) or rayPrimary.rmiss.glsl:40-106 (misses), followed by Russian
// roulette (russian_roulette.glsl:1-11).
// One kernel per material-sorted queue (k_partition): KIND 0 shades the
// Lambert hits, 1 the metallic/roughness hits, 2 the misses. Each is compiled
// for its own case only (the other surface models are dead code there), so
// the Lambert and miss kernels fit more resident blocks than the
// metallic/roughness one.
// VVPT_SHADE_SHARED_BSDF: one call site for the cosine-weighted warp and one
// copy of the metallic/roughness evaluation in the surface event.
#ifndef VVPT_SHADE_SHARED_BSDF
#define VVPT_SHADE_SHARED_BSDF 1
#endif
template <int KIND, bool kOne>
__global__ void __launch_bounds__(256, KIND == 0 || KIND == 2 ? VVPT_SHADE_LM_MIN_BLOCKS : VVPT_SHADE_MIN_BLOCKS)
    k_shade(JobTable jt, PathState ps, Queues q, int pp, const __grid_constant__ JobView one)
{
    // KIND 3: all three queues in one launch (VVPT_SHADE_SPLIT = 0)
    const uint32_t nl = q.counters[C_SHADE_L], np = q.counters[C_SHADE_P];
    const uint32_t n = KIND == 3 ? nl + np + q.counters[C_SHADE_M]
                                 : q.counters[KIND == 0 ? C_SHADE_L : (KIND == 1 ? C_SHADE_P : C_SHADE_M)];
    const uint32_t *queue = KIND == 0 ? q.shade_l : (KIND == 1 ? q.shade_p : q.shade_m);
    auto entry = [&](uint32_t i) {
        if (KIND != 3)
            return queue[i];
        return i < nl ? q.shade_l[i] : (i < nl + np ? q.shade_p[i - nl] : q.shade_m[i - nl - np]);
    };
    uint32_t err = 0, walks = 0;
    {
        const uint32_t f = blockIdx.x * blockDim.x;
        if (f < n)
            tlas_cache_fill(job_view<kOne>(jt, one, ps[entry(f)].job).scene);
        else
            tlas_cache_none();
    }
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t slot = 0;
        bool want_conn = false, want_nee = false, want_done = false, want_ext = false;
        bool late = false; // an ended path with a ray still to trace: regen runs after it, an iteration later
        if (i < n) {
        slot = entry(i);
        float4 hv, mv, bv, rv, ov, dv;
        load_pair(ps[slot].hit, hv, mv);
        load_pair(ps[slot].beta, bv, rv);
        load_pair(ps[slot].o, ov, dv);
        const JobView &J = job_view<kOne>(jt, one, __float_as_uint(mv.z));
        const SceneView &s = J.scene;
        const RenderParams &p = J.params;

        uint32_t flags = __float_as_uint(mv.x);
        PathRng rng = load_rng(p, ps, slot, __float_as_uint(bv.w));
        float3 beta = f3(bv);
        float3 rad = f3(rv);
        if (flags & F_NEE) // the previous event's emitter ray (a path that continued with zfar > kExtTmax)
            rad = rad + f3(ps[slot].nee_c);
        float3 origin = f3(ov);
        float3 dir = f3(dv);
        uint32_t vol = __float_as_uint(mv.y);
        const uint32_t d = (flags >> kDepthShift) & kByteMask;
        uint32_t sdepth = (flags >> kSurfShift) & kByteMask;
        bool inside = (flags & F_INSIDE) != 0;
        const uint32_t inst_id = __float_as_uint(mv.w);
        const bool is_hit = KIND == 3 ? inst_id != kNoHit : KIND != 2; // hits (0, 1) or misses (2)

        // the previous event's emitter ray, added before this event's own
        // contributions (next_event_estimation.glsl:28-32 runs inside the
        // previous hit shader)
        if (flags & F_NEE_FUSED)
            rad += fused_nee(s, p, (flags & F_NEE_FULL) != 0, is_hit, inst_id, hv, origin, dir, inside, vol,
                             ps[slot].nee_b, err, walks);

        bool stop = false;
        bool terminal_no_rr = false; // returns before the RR block
        bool has_shadow = false, has_nee = false;
        bool sampled = false;        // a new direction was sampled here (pdf in nee_pdf)
        bool keep_sampled = false;   // pass-through: the direction keeps its sampling pdf
        const bool last = (d + 1u >= p.depth);
        float3 sh_dir = f3(0.0f), sh_c = f3(0.0f);
        float sh_tmax = 0.0f;
        float3 nee_beta = f3(0.0f);
        float nee_pdf = 0.0f;
        bool write_alb = false;
        float3 new_alb = f3(0.0f), new_nrm = f3(0.0f);

        // ---- medium along the segment
        bool sampled_medium = false;
        float3 scatter_pos = f3(0.0f);
        float g = 0.0f;
        if (inside && vol < s.num_materials) {
            float vtend = is_hit ? hv.x : fminf(p.zfar_trunc, kExtTmax);
            sampled_medium = medium_event(s, p, vol, kExtTmin, vtend, origin, dir, beta, rng, scatter_pos, g);
        }
        // The event's own part first; an event that samples a light (a
        // scatter point in a medium, or a surface the path continues from)
        // then samples it at one call site, so that the light-sampling code
        // (mesh lights, environment) is inlined once; the evaluation after it
        // follows per event. The random numbers are drawn in the same order.
        SurfaceHit h;
        bool lambert = false, surface_light = false;
        float3 albedo = f3(0.0f);
        PBR pbr;
        if (sampled_medium) {
            // light sample at the scatter point with the HG phase function
            // (process_volume_hit.glsl:42-79), below
        } else if (!is_hit) {
            // miss: background (rayPrimary.rmiss.glsl:53-103)
            stop = true;
            terminal_no_rr = true;
            const int mode = (int)p.env_type;
            // with the environment light-sampled, a sampled direction's escape
            // takes the BSDF side of the MIS weight
            float wenv = 1.0f;
            if (p.env_light && (flags & F_SAMPLED))
                wenv = power_heuristic(ps[slot].nee_b.w, env_pdf(s, dir) / (float)(p.num_lights + 1u));
            // one environment lookup for modes 1 and 2 (one inlined copy)
            const bool env_seen = mode == 1 || (mode == 2 && sdepth != 0);
            const float3 envc = env_seen ? env_lookup(s, dir) : f3(0.0f);
            if (mode == 0) {
                if (sdepth == 0) {
                    write_alb = true;
                    new_alb = p.background;
                    new_nrm = f3(0.0f);
                }
                rad += p.background * beta;
            } else if (mode == 1) {
                float3 bg = p.env_intensity * envc;
                if (sdepth == 0) {
                    write_alb = true;
                    new_alb = bg;
                    new_nrm = f3(0.0f);
                }
                rad += bg * beta * wenv;
            } else if (mode == 2) {
                if (sdepth == 0) {
                    write_alb = true;
                    new_alb = p.background;
                    new_nrm = f3(0.0f);
                    rad += p.background * beta;
                } else {
                    rad += envc * beta * wenv;
                }
            }
        } else {
            // surface event
            const uint32_t prim = __float_as_uint(hv.w);
            h = make_surface_hit(s, inst_id, prim, hv.y, hv.z, dir);
            const DevMaterial &m = s.materials[h.material];
            const float2 tuv = make_float2(h.uv.x * m.uv_tiling.x, h.uv.y * m.uv_tiling.y);
            lambert = KIND == 3 ? (uint32_t)m.uv_tiling.z == 2u : KIND == 0;
            bool passthrough = false;
            if (m.mrao.w > 0.0f) {
                float alpha = material_alpha(s, m, tuv);
                float r = rnd1(p, rng);
                if (alpha < kEps || r > alpha) {
                    if (h.front_volume != h.back_volume) {
                        inside = false;
                        int nv = h.flipped ? h.front_volume : h.back_volume;
                        if (nv != -1) {
                            inside = true;
                            vol = (uint32_t)nv;
                        }
                    }
                    origin = h.wpos;
                    dir = normalize3(dir);
                    passthrough = true;
                    keep_sampled = (flags & F_SAMPLED) != 0;
                }
            }
            if (passthrough) {
                terminal_no_rr = true; // returns without RR and without stop
            } else {
                float4 nm = tex2d(s, m.tex2[1], tuv.x, tuv.y);
                apply_normal_to_frame(h.frame, normal_from_normal_map(f3(nm)));
                albedo = f3(m.albedo) * f3(tex2d(s, m.tex1[0], tuv.x, tuv.y));
                float3 emissive = material_emissive(s, m, tuv);
                if (!lambert) {
                    pbr.albedo = albedo;
                    pbr.metallic = m.mrao.x * tex2d(s, m.tex1[1], tuv.x, tuv.y).x;
                    pbr.roughness = m.mrao.y * tex2d(s, m.tex1[2], tuv.x, tuv.y).x;
                    pbr.roughness = fmaxf(pbr.roughness, 0.035f);
                }
                if (sdepth == 0) {
                    write_alb = true;
                    new_alb = albedo;
                    new_nrm = h.frame.n * 0.5f + f3(0.5f);
                }
                const float em_eps = lambert ? 0.05f : 0.1f;
                if (sdepth == 0 && !is_black_eps(emissive, em_eps) && !h.flipped) {
                    rad += emissive * beta;
                    stop = true;
                    terminal_no_rr = true;
                } else {
                    sdepth = min(sdepth + 1u, 255u);
                    surface_light = true;
                }
            }
        }
        if (sampled_medium || surface_light) {
            // in background mode 2 an escape before any surface event sees
            // the solid colour, so the environment is not a light there
            const LightSample ls =
                sample_light(s, p, sampled_medium ? scatter_pos : h.wpos, rng,
                             sampled_medium ? !last && !((int)p.env_type == 2 && sdepth == 0) : !last);
            if (sampled_medium) {
                float3 wo = -normalize3(dir);
                if (!is_black(ls.radiance)) {
                    float ph = henyey_greenstein(dot3(wo, ls.dir), g);
                    float3 F = f3(ph);
                    if (!is_black(F)) {
                        float w = ls.delta ? 1.0f : power_heuristic(ls.pdf, ph);
                        has_shadow = true;
                        sh_dir = ls.dir;
                        sh_tmax = ls.tmax;
                        sh_c = (ls.delta ? ls.radiance : w * ls.radiance) * F * beta / ls.pdf;
                    }
                }
                float3 wi;
                const float2 uu = rnd2(p, rng);
                const float u0 = uu.x, u1 = uu.y;
                float spdf = hg_sample(wo, wi, u0, u1, g);
                origin = scatter_pos;
                dir = wi;
                has_nee = true;
                sampled = true;
                nee_beta = beta;
                nee_pdf = spdf;
            } else {
                const float3 wo = world_to_local(h.frame, -dir);
#if VVPT_SHADE_SHARED_BSDF
                // The BSDF sample's numbers follow the light sample's, as
                // always; the cosine-weighted warp serves Lambert surfaces
                // and the metallic/roughness diffuse lobe from one call site,
                // and one copy of the metallic/roughness evaluation (a loop
                // that is not unrolled) takes the light's direction and the
                // sampled one. Same arithmetic as sample_pbr.
                const float2 uu = rnd2(p, rng);
                const float rl = lambert ? 0.0f : rnd1(p, rng);
                float spdf = 0.0f;
                float3 sdir_local;
                if (lambert || rl <= diffuse_sampling_ratio(pbr))
                    sdir_local = cosine_sample_hemisphere(uu.x, uu.y, spdf);
                else
                    sdir_local = ggx_sample_reflect(wo, pbr, uu.x, uu.y);
                const float3 wil = world_to_local(h.frame, ls.dir);
                float3 Fl = f3(0.0f), Fsm = f3(0.0f);
                float pl = 0.0f, psm = 0.0f;
                if (lambert) {
                    const float ct = fminf(fmaxf(wil.y, 0.0f), 1.0f);
                    Fl = albedo * kInvPi * ct;
                    pl = cosine_hemisphere_pdf(ct);
                } else {
#pragma unroll 1
                    for (int k = 0; k < 2; k++) {
                        const float3 wi = k == 0 ? wil : sdir_local;
                        const float3 F = eval_pbr(pbr, wi, wo, normalize3(wo + wi));
                        const float pd = pdf_pbr(wi, wo, pbr);
                        if (k == 0) {
                            Fl = F;
                            pl = ls.delta ? 0.0f : pd;
                        } else {
                            Fsm = F;
                            psm = pd;
                        }
                    }
                }
                if (!is_black(ls.radiance) && !is_black(Fl)) {
                    float w = ls.delta ? 1.0f : power_heuristic(ls.pdf, pl);
                    has_shadow = true;
                    sh_dir = ls.dir;
                    sh_tmax = ls.tmax;
                    sh_c = (ls.delta ? ls.radiance : w * ls.radiance) * Fl * beta / ls.pdf;
                }
                bool black_f = false;
                float3 Fs = f3(0.0f);
                if (!lambert) {
                    spdf = psm;
                    Fs = psm < kEps ? f3(0.0f) : Fsm;
                    black_f = is_black(Fs);
                }
#else
                if (!is_black(ls.radiance)) {
                    float3 wi = world_to_local(h.frame, ls.dir);
                    float3 F;
                    float bpdf;
                    if (lambert) {
                        float ct = fminf(fmaxf(wi.y, 0.0f), 1.0f);
                        F = albedo * kInvPi * ct;
                        bpdf = cosine_hemisphere_pdf(ct);
                    } else {
                        F = eval_pbr(pbr, wi, wo, normalize3(wo + wi));
                        bpdf = ls.delta ? 0.0f : pdf_pbr(wi, wo, pbr);
                    }
                    if (!is_black(F)) {
                        float w = ls.delta ? 1.0f : power_heuristic(ls.pdf, bpdf);
                        has_shadow = true;
                        sh_dir = ls.dir;
                        sh_tmax = ls.tmax;
                        sh_c = (ls.delta ? ls.radiance : w * ls.radiance) * F * beta / ls.pdf;
                    }
                }
                // BSDF sampling
                float spdf;
                float3 sdir_local;
                bool black_f = false;
                float3 Fs;
                if (lambert) {
                    const float2 uu = rnd2(p, rng);
                    const float u0 = uu.x, u1 = uu.y;
                    sdir_local = cosine_sample_hemisphere(u0, u1, spdf);
                } else {
                    const float2 uu = rnd2(p, rng);
                    const float u0 = uu.x, u1 = uu.y;
                    float r = rnd1(p, rng);
                    Fs = sample_pbr(sdir_local, wo, spdf, pbr, u0, u1, r);
                    black_f = is_black(Fs);
                }
#endif
                float3 sdir = local_to_world(h.frame, sdir_local);
                origin = h.wpos;
                dir = sdir;
                if (lambert) {
                    beta *= albedo;
                    has_nee = true;
                } else if (black_f) {
                    stop = true;
                    terminal_no_rr = true;
                } else {
                    beta *= clamp3(Fs / spdf, 0.0f, 1.0f);
                    has_nee = true;
                }
                sampled = has_nee;
                nee_beta = beta;
                nee_pdf = spdf;
            }
        }
        // Russian roulette (russian_roulette.glsl:1-11) for events that reach it
        if (!terminal_no_rr) {
            float rr = rnd1(p, rng);
            if (d > kRussianRouletteDepth) {
                float mb = fmaxf(beta.x, fmaxf(beta.y, beta.z));
                if (rr >= mb)
                    stop = true;
                else
                    beta = beta * (1.0f / mb);
            }
        }
        if (has_nee && p.num_lights == 0u) {
            // With no lights the reference's emitter pdf is
            // lightDirectPdf * (1 / 0) = inf (rayNEE.rahit.glsl:124), so the
            // MIS weight and the contribution are zero: skip the ray.
            has_nee = false;
        }
        if (has_nee && !may_reach_emitter(s, origin, dir))
            has_nee = false; // no emissive surface on its line: it adds zero

        const bool done = stop || last;
        uint32_t nf = F_ITEM | (inside ? F_INSIDE : 0u) | ((min(d + 1u, 255u)) << kDepthShift) | (sdepth << kSurfShift);
        if (done)
            nf |= F_DONE;
        if (has_shadow)
            nf |= F_SHADOW;
        if (sampled || keep_sampled)
            nf |= F_SAMPLED;
        // a continuing path's emitter ray shares origin and direction with its
        // next extension ray and is resolved from that traversal
        const bool fuse = has_nee && !done && p.zfar <= kExtTmax;
        if (has_nee)
            nf |= fuse ? F_NEE_FUSED : F_NEE;
        *reinterpret_cast<uint2 *>(&ps[slot].flags) = make_uint2(nf, vol);
        store_pair(ps[slot].beta, f4(beta, __uint_as_float(rng.s)), f4(rad, 0.0f));
        store_pair(ps[slot].o, f4(origin, 0.0f), f4(dir, 0.0f));
        if (write_alb)
            store_pair(ps[slot].alb, f4(new_alb, 0.0f), f4(new_nrm, 0.0f));
        if (has_shadow)
            store_pair(ps[slot].sh_dir, f4(sh_dir, sh_tmax), f4(sh_c, 0.0f));
        if (sampled)
            ps[slot].nee_b = f4(nee_beta, nee_pdf);
        want_conn = has_shadow;
        want_nee = has_nee && !fuse;
        want_done = done;
        late = want_conn || want_nee;
        want_ext = !done;
        }
        const bool now = want_done && !late, later = want_done && late;
        uint32_t pos[5];
        warp_append_many<5>({want_ext, want_conn, now, later, want_nee},
                            {&q.counters[C_EXT0 + (1 - pp)], &q.counters[C_CONN], &q.counters[C_REGEN0 + (1 - pp)],
                             &q.counters[C_REGEN0 + pp], &q.counters[C_NEEQ]},
                            pos);
        if (want_ext)
            q.ext[1 - pp][pos[0]] = slot;
        if (want_conn)
            q.conn[pos[1]] = slot;
        if (now)
            q.regen[1 - pp][pos[2]] = slot;
        if (later)
            q.regen[pp][pos[3]] = slot;
        if (want_nee)
            q.nee[pos[4]] = slot;
    }
    warp_add(&q.counters[C_NEE], walks);
    if (err)
        atomicOr(&q.counters[C_ERR], err);
}

// Shadow ray with transparent surfaces and media (lightSampling.glsl:108-144,
// raySecondary.rahit.glsl:31-72, raySecondary.rchit.glsl:32-78,
// raySecondary.rmiss.glsl:17-44). Candidates are processed nearest first.
__device__ float3 shadow_transmittance(const SceneView &s, const RenderParams &p, float3 o,
                                       const float3 &dir, float tmax_light, bool inside, uint32_t vol, uint32_t &err)
{
    const float tmin = kConnTmin;
    float3 T = f3(1.0f);
    bool shadowed = false;
    bool stop = false;
    float distT = tmax_light - tmin;
    for (uint32_t seg = 0; seg < p.depth; seg++) {
        float vtmin = tmin;
        Hit after = no_hit();
        bool accepted = false;
        Hit acc;
        int guard = 0;
        for (;;) {
            Hit h = trace_after(s, o, dir, tmin, distT, after, err);
            if (h.inst == kNoHit)
                break;
            if (++guard > kCandidateCap) {
                err |= kErrLoopCap;
                stop = shadowed = true;
                accepted = true;
                acc = h;
                break;
            }
            const DevInstance &inst = s.instances[h.inst];
            const DevMaterial &m = s.materials[inst.material];
            if (!(m.mrao.w >= 0.99f)) {
                stop = shadowed = true;
                accepted = true;
                acc = h;
                break;
            }
            // alpha needs the hit's uv
            ShadeVertex a, b, c;
            fetch_triangle(s, inst, h.prim, a, b, c);
            float bx = 1.0f - h.u - h.v;
            float2 uv = make_float2(a.pos_u.w * bx + b.pos_u.w * h.u + c.pos_u.w * h.v,
                                    a.nrm_v.w * bx + b.nrm_v.w * h.u + c.nrm_v.w * h.v);
            float alpha = material_alpha(s, m, make_float2(uv.x * m.uv_tiling.x, uv.y * m.uv_tiling.y));
            T *= f3(1.0f - alpha);
            if (inst.front_volume != inst.back_volume) {
                accepted = true;
                acc = h;
                break;
            }
            if (max3f(T) > kEps) {
                shadowed = false;
                after = h;
                continue;
            }
            stop = shadowed = true;
            accepted = true;
            acc = h;
            break;
        }
        if (!accepted) {
            // miss shader
            stop = true;
            shadowed = false;
            if (inside && vol < s.num_materials) {
                float vtend = fminf(p.zfar_trunc, distT);
                T *= medium_transmittance(s, vol, vtmin, vtend);
                shadowed = !(max3f(T) > kEps);
            }
        } else if (!stop) {
            // closest hit on a volume boundary
            SurfaceHit sh = make_surface_hit(s, acc.inst, acc.prim, acc.u, acc.v, dir);
            bool ended = false;
            if (inside && vol < s.num_materials) {
                T *= medium_transmittance(s, vol, vtmin, acc.t);
                if (max3f(T) < kEps) {
                    stop = shadowed = true;
                    ended = true;
                }
            }
            if (!ended) {
                vtmin = acc.t;
                inside = false;
                int nv = sh.flipped ? sh.front_volume : sh.back_volume;
                if (nv != -1) {
                    inside = true;
                    vol = (uint32_t)nv;
                }
                o = sh.wpos;
            }
        }
        distT -= vtmin;
        if (stop)
            break;
    }
    if (shadowed)
        T = f3(0.0f);
    return T;
}

// An emitter reached by the BSDF-direction ray (rayNEE.rahit.glsl:73-131):
// medium transmittance up to the hit, back-face rejection, and the light pdf
// of having sampled that point, with the squared distance measured from the
// object-space ray origin as the reference does (rayNEE.rahit.glsl:122).
__device__ __forceinline__ void emitter_eval(const SceneView &s, const RenderParams &p, const DevInstance &inst,
                                             const ShadeVertex &a, const ShadeVertex &b, const ShadeVertex &c,
                                             const Hit &h, const float3 &e, const float3 &o, const float3 &dir,
                                             bool inside, uint32_t vol, float vtmin, float3 &T, float3 &em, float &pdf)
{
    if (inside && vol < s.num_materials) {
        T *= medium_transmittance(s, vol, vtmin, h.t);
        if (max3f(T) < kEps) {
            T = f3(0.0f);
            em = f3(0.0f);
            return;
        }
    }
    const float bx = 1.0f - h.u - h.v;
    Affine34 w2o = rows_of(inst.w2o), o2w = rows_of(inst.o2w);
    float3 ln = f3(a.nrm_v) * bx + f3(b.nrm_v) * h.u + f3(c.nrm_v) * h.v;
    float3 wn = normalize3(xform_normal_transposed(w2o, ln));
    if (dot3(wn, dir) > 0.0f) { // back face
        em = f3(0.0f);
        T = f3(0.0f);
        return;
    }
    em = e;
    float3 lp = f3(a.pos_u) * bx + f3(b.pos_u) * h.u + f3(c.pos_u) * h.v;
    float3 wp = xform_point(o2w, lp);
    float3 p0 = xform_point(o2w, f3(a.pos_u)), p1 = xform_point(o2w, f3(b.pos_u)), p2 = xform_point(o2w, f3(c.pos_u));
    float area = 0.5f * length3(cross3(p1 - p0, p2 - p0));
    float point_pdf = (1.0f / (float)inst.num_triangles) * (1.0f / area);
    float dp = dot3(-dir, wn);
    if (dp > 0.0f) {
        float3 obj_o = xform_point(w2o, o);
        float dist = length3(obj_o - wp);
        float light_pdf = point_pdf * (dist * dist) / dp;
        pdf = light_pdf * (1.0f / (float)(p.num_lights + p.env_light));
    } else {
        pdf = 0.0f;
        em = f3(0.0f);
    }
}

// BSDF-direction emitter ray (next_event_estimation.glsl:1-33,
// rayNEE.rahit.glsl:32-132, rayNEE.rchit.glsl:33-82, rayNEE.rmiss.glsl:12-19).
// Returns the emitter radiance times throughput and its light pdf.
__device__ __noinline__ void emitter_ray(const SceneView &s, const RenderParams &p, float3 o,
                                         const float3 &dir, bool inside, uint32_t vol, float3 &out_em_T,
                                         float3 &out_T, float3 &out_em, float &out_pdf, uint32_t &err)
{
    const float tmin = kConnTmin;
    const float tmax = p.zfar;
    float3 T = f3(1.0f);
    float3 em = f3(0.0f);
    float pdf = 0.0f;
    bool stop = false;
    for (uint32_t seg = 0; seg < p.depth; seg++) {
        float vtmin = tmin;
        Hit after = no_hit();
        bool accepted = false;
        Hit acc;
        int guard = 0;
        for (;;) {
            Hit h = trace_after(s, o, dir, tmin, tmax, after, err);
            if (h.inst == kNoHit)
                break;
            if (++guard > kCandidateCap) {
                err |= kErrLoopCap;
                stop = true;
                T = f3(0.0f);
                em = f3(0.0f);
                accepted = true;
                acc = h;
                break;
            }
            const DevInstance &inst = s.instances[h.inst];
            const DevMaterial &m = s.materials[inst.material];
            ShadeVertex a, b, c;
            fetch_triangle(s, inst, h.prim, a, b, c);
            float bx = 1.0f - h.u - h.v;
            float2 uv = make_float2(a.pos_u.w * bx + b.pos_u.w * h.u + c.pos_u.w * h.v,
                                    a.nrm_v.w * bx + b.nrm_v.w * h.u + c.nrm_v.w * h.v);
            float2 tuv = make_float2(uv.x * m.uv_tiling.x, uv.y * m.uv_tiling.y);
            float3 e = material_emissive(s, m, tuv);
            const bool transparent = m.mrao.w >= 0.99f;
            if (is_black_eps(e, 0.05f)) {
                if (!transparent) {
                    stop = true;
                    T = f3(0.0f);
                    em = f3(0.0f);
                    accepted = true;
                    acc = h;
                    break;
                }
                float alpha = material_alpha(s, m, tuv);
                T *= f3(1.0f - alpha);
                if (inst.front_volume != inst.back_volume) {
                    accepted = true;
                    acc = h;
                    break;
                }
                after = h;
                continue;
            }
            // emissive surface
            stop = true;
            accepted = true;
            acc = h;
            emitter_eval(s, p, inst, a, b, c, h, e, o, dir, inside, vol, vtmin, T, em, pdf);
            break;
        }
        if (!accepted) {
            stop = true;
            em = f3(0.0f);
            pdf = 0.0f;
        } else if (!stop) {
            SurfaceHit sh = make_surface_hit(s, acc.inst, acc.prim, acc.u, acc.v, dir);
            bool ended = false;
            if (inside && vol < s.num_materials) {
                T *= medium_transmittance(s, vol, vtmin, acc.t);
                if (max3f(T) < kEps) {
                    stop = true;
                    T = f3(0.0f);
                    em = f3(0.0f);
                    ended = true;
                }
            }
            if (!ended) {
                vtmin = acc.t;
                inside = false;
                int nv = sh.flipped ? sh.front_volume : sh.back_volume;
                if (nv != -1) {
                    inside = true;
                    vol = (uint32_t)nv;
                }
                o = sh.wpos;
            }
        }
        if (stop)
            break;
    }
    out_T = T;
    out_em = em;
    out_pdf = pdf;
    out_em_T = T * em;
}

// The BSDF-direction emitter ray from its first candidate (the closest hit
// along the ray from the emitter ray's tmin): true when that candidate is
// transparent and the complete candidate walk of emitter_ray is needed,
// otherwise T, em and pdf are the ray's. No candidate, or one beyond zfar, is
// a miss.
__device__ __forceinline__ bool emitter_first(const SceneView &s, const RenderParams &p, bool is_hit, uint32_t inst_id,
                                              const float4 &hv, const float3 &o, const float3 &dir, bool inside,
                                              uint32_t vol, float3 &T, float3 &em, float &pdf)
{
    if (!is_hit || !(hv.x <= p.zfar))
        return false;
    Hit h;
    h.t = hv.x;
    h.u = hv.y;
    h.v = hv.z;
    h.inst = inst_id;
    h.prim = __float_as_uint(hv.w);
    const DevInstance &inst = s.instances[inst_id];
    const DevMaterial &m = s.materials[inst.material];
    ShadeVertex a, b, c;
    fetch_triangle(s, inst, h.prim, a, b, c);
    const float bx = 1.0f - h.u - h.v;
    float2 uv = make_float2(a.pos_u.w * bx + b.pos_u.w * h.u + c.pos_u.w * h.v,
                            a.nrm_v.w * bx + b.nrm_v.w * h.u + c.nrm_v.w * h.v);
    float2 tuv = make_float2(uv.x * m.uv_tiling.x, uv.y * m.uv_tiling.y);
    float3 e = material_emissive(s, m, tuv);
    if (is_black_eps(e, 0.05f))
        return m.mrao.w >= 0.99f; // transparent: walk the candidates
    emitter_eval(s, p, inst, a, b, c, h, e, o, dir, inside, vol, kConnTmin, T, em, pdf);
    return false;
}

// The previous event's BSDF-direction emitter ray, resolved from this
// iteration's extension hit: the two rays share origin and direction, and the
// extension traversal starts at the emitter ray's tmin (1e-4) when one is
// pending, so the extension hit is the emitter ray's first candidate unless
// extend flagged a candidate below 1e-3 (`full`).
__device__ __noinline__ float3 fused_nee(const SceneView &s, const RenderParams &p, bool full, bool is_hit,
                                         uint32_t inst_id, float4 hv, float3 o, float3 dir, bool inside, uint32_t vol,
                                         float4 nb, uint32_t &err, uint32_t &walks)
{
    float3 T = f3(1.0f), em = f3(0.0f);
    float pdf = 0.0f;
    if (full || emitter_first(s, p, is_hit, inst_id, hv, o, dir, inside, vol, T, em, pdf)) {
        float3 emT;
        emitter_ray(s, p, o, dir, inside, vol, emT, T, em, pdf, err);
        walks++;
    }
    if (is_black(em))
        return f3(0.0f);
    return power_heuristic(nb.w, pdf) * T * em * f3(nb);
}

// The rays that need the full any-hit candidate walk, one lane each, before
// shade adds this iteration's contributions: shadow rays whose nearest
// candidate is transparent and fused emitter rays whose first candidate is
// transparent or below the extension ray's tmin (one queue entry per path, the
// shadow ray's contribution first, in the order of the reference's
// additions), then the emitter rays traced on their own. Those of ended paths
// have their first candidate from k_trace and walk only past a transparent
// one. They write their contribution to nee_c, so the two parts never write
// the same word; regen (or shade, for a path that continues) adds it after
// the shadow ray's.
__global__ void __launch_bounds__(256, VVPT_WALK_MIN_BLOCKS) k_walk(JobTable jt, PathState ps, Queues q)
{
    const uint32_t nw = q.counters[C_WALK];
    const uint32_t n = nw + q.counters[C_NEE_RUN];
    uint32_t err = 0, nnee = 0;
    // a short queue (the usual case) is spread over the grid's warps, so that
    // few walks, or only one, share a warp and none waits for another's steps
    // (1920 x 1080 x 32 medium scene, about 2300 entries a launch: 106 us a
    // launch with 32 to a warp, 56 us spread)
    uint32_t spread = 1;
    while (spread < 32u && (unsigned long long)n * (2u * spread) <= gridDim.x * blockDim.x)
        spread *= 2u;
    const uint32_t b0 = first_ray() / spread;
    if (b0 < n)
        tlas_cache_fill(jt.jobs[ps[b0 < nw ? q.walk[b0] : q.nee[b0 - nw]].job].scene);
    else
        tlas_cache_none();
    for (uint32_t i = my_ray() % spread ? n : my_ray() / spread; i < n; i += ray_stride() / spread) {
        const uint32_t slot = i < nw ? q.walk[i] : q.nee[i - nw];
        const JobView &J = jt.jobs[ps[slot].job];
        const SceneView &s = J.scene;
        const RenderParams &p = J.params;
        const uint32_t flags = ps[slot].flags; // of an emitter ray's entry only F_INSIDE: the other part may write the rest
        const bool inside = (flags & F_INSIDE) != 0;
        if (i < nw && (flags & F_SHADOW_WALK)) {
            const float4 sd = ps[slot].sh_dir;
            const float3 T = shadow_transmittance(s, p, f3(ps[slot].o), f3(sd), sd.w, inside, ps[slot].vol, err);
            if (!is_black(T))
                ps[slot].rad = f4(f3(ps[slot].rad) + f3(ps[slot].sh_c) * T, 0.0f);
        }
        if (i >= nw || (flags & F_NEE_FULL)) {
            const float4 nb = ps[slot].nee_b;
            const float3 o = f3(ps[slot].o), d = f3(ps[slot].d);
            const uint32_t vol = ps[slot].vol;
            float3 emT, T = f3(1.0f), em = f3(0.0f);
            float lpdf = 0.0f;
            const uint32_t inst = ps[slot].hit_inst;
            if (i < nw || !(flags & F_DONE) ||
                emitter_first(s, p, inst != kNoHit, inst, ps[slot].hit, o, d, inside, vol, T, em, lpdf))
                emitter_ray(s, p, o, d, inside, vol, emT, T, em, lpdf, err);
            nnee++;
            if (i < nw) {
                if (!is_black(em))
                    ps[slot].rad = f4(f3(ps[slot].rad) + power_heuristic(nb.w, lpdf) * T * em * f3(nb), 0.0f);
                ps[slot].flags = flags & ~(F_NEE_FUSED | F_NEE_FULL | F_SHADOW_WALK);
            } else {
                float3 c = f3(0.0f);
                if (!is_black(em))
                    c = power_heuristic(nb.w, lpdf) * T * em * f3(nb);
                ps[slot].nee_c = f4(c, 0.0f);
            }
        }
    }
    warp_add(&q.counters[C_NEE], nnee);
    if (err)
        atomicOr(&q.counters[C_ERR], err);
}

// Final image: per pixel, add the per-batch sums in batch order starting from
// zero, exactly the sequence of read-modify-writes of raygen.rgen.glsl:134-144.
__global__ void k_reduce(RenderParams p, BatchResults br, float4 *rad, float4 *alb, float4 *nrm, float4 *m2)
{
    const uint32_t npix = p.width * p.height;
    for (uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x; pix < npix; pix += gridDim.x * blockDim.x) {
        float3 r = f3(0.0f), a = f3(0.0f), nn = f3(0.0f), q2 = f3(0.0f);
        if (p.reduce_fp64) {
            double s[12] = {0.0};
            for (uint32_t b = 0; b < p.batches; b++) {
                const size_t it = (size_t)b * npix + pix;
                const float4 rb = br.rad[it], ab = br.alb[it], nb = br.nrm[it];
                s[0] += rb.x, s[1] += rb.y, s[2] += rb.z;
                s[3] += ab.x, s[4] += ab.y, s[5] += ab.z;
                s[6] += nb.x, s[7] += nb.y, s[8] += nb.z;
                s[9] += (double)rb.x * rb.x, s[10] += (double)rb.y * rb.y, s[11] += (double)rb.z * rb.z;
            }
            r = f3((float)s[0], (float)s[1], (float)s[2]);
            a = f3((float)s[3], (float)s[4], (float)s[5]);
            nn = f3((float)s[6], (float)s[7], (float)s[8]);
            q2 = f3((float)s[9], (float)s[10], (float)s[11]);
        } else {
            for (uint32_t b = 0; b < p.batches; b++) {
                const size_t it = (size_t)b * npix + pix;
                float3 rb = f3(br.rad[it]);
                r = r + rb;
                a = a + f3(br.alb[it]);
                nn = nn + f3(br.nrm[it]);
                q2 = q2 + rb * rb;
            }
        }
        if (rad)
            rad[pix] = f4(r, 1.0f);
        if (alb)
            alb[pix] = f4(a, 1.0f);
        if (nrm)
            nrm[pix] = f4(nn, 1.0f);
        if (m2)
            m2[pix] = f4(q2, 1.0f);
    }
}

// Closest hits of a caller's rays, written in the caller's layout (20 bytes).
// One ray per lane: for as many rays as the refill form below has lanes, where
// there is nothing to refill (100,000 rays: 42 us, 58 with the refill loop).
__global__ void k_trace_closest(SceneView s, const float4 *rays, uint32_t n, vvpt_hit *hits, uint32_t *status)
{
    uint32_t err = 0;
    tlas_cache_fill(s);
    for (uint32_t i = my_ray(); i < n; i += ray_stride()) {
        const float4 a = rays[2 * (size_t)i], b = rays[2 * (size_t)i + 1];
        const Hit h = trace_closest(s, f3(a), f3(b), a.w, b.w, err);
        hits[i] = vvpt_hit{h.t, h.u, h.v, h.inst, h.prim};
    }
    if (err)
        atomicOr(&status[0], err);
}

// The same with k_trace's lane refill (a million rays, half of them incoherent:
// 0.52 ms one ray per lane, 0.40 ms here). status[0]: error bits, status[1]:
// rays handed out.
__global__ void __launch_bounds__(256, VVPT_TRACE_MIN_BLOCKS) k_trace_closest_refill(SceneView s, const float4 *rays, uint32_t n,
                                                                              vvpt_hit *hits, uint32_t *status)
{
    uint32_t err = 0;
    tlas_cache_fill(s);
    __shared__ uint32_t cold_i[256];
    __shared__ float4 cold_o[256], cold_d[256], cold_best[256];
    __shared__ uint2 cold_ids[256];
    const TraceCold ray{cold_o[threadIdx.x], cold_d[threadIdx.x], cold_best[threadIdx.x], cold_ids[threadIdx.x]};
    TraceState st;
    TraceStack stack;
    uint32_t state = kLaneFree;
    bool open = true;
    for (;;) {
        uint32_t tr = __ballot_sync(0xFFFFFFFFu, state == kLaneTracing);
        if (__popc(tr) <= (open ? VVPT_REFILL_BELOW : 0)) {
            if (state == kLaneDone) {
                const Hit h = trace_best(ray);
                hits[cold_i[threadIdx.x]] = vvpt_hit{h.t, h.u, h.v, h.inst, h.prim};
                state = kLaneFree;
            }
            if (open) {
                bool mine;
                const uint32_t i = refill_take(state == kLaneFree, &status[1], n, open, mine);
                if (mine) {
                    const float4 a = rays[2 * (size_t)i], b = rays[2 * (size_t)i + 1];
                    cold_i[threadIdx.x] = i;
                    trace_begin(st, ray, s, f3(a), f3(b), a.w, b.w, no_hit());
                    state = kLaneTracing;
                }
            }
            tr = __ballot_sync(0xFFFFFFFFu, state == kLaneTracing);
            if (tr == 0) {
                if (!open)
                    break;
                continue;
            }
        }
        if (trace_turn(st, ray, stack, s, state == kLaneTracing, __popc(tr), err))
            state = kLaneDone;
    }
    if (err)
        atomicOr(&status[0], err);
}

// ---------------------------------------------------------------------------
// Host launchers

void launch_init_slots(const Queues &q, const PathState &ps, const JobTable &jt, uint32_t slots, cudaStream_t stream)
{
    int grid = (int)std::min<uint32_t>((slots + 255) / 256, 65535u);
    k_init_slots<<<grid, 256, 0, stream>>>(q, ps, jt, slots);
}

void launch_admit(const Queues &q, const JobTable &jt, unsigned long long total_items, uint32_t num_ranges,
                  cudaStream_t stream)
{
    k_admit<<<1, 1024, 0, stream>>>(q, jt, total_items, num_ranges);
}

void launch_iteration(const JobTable &jt, const PathState &ps, const Queues &q, int pp, const LaunchShape &shape,
                      cudaStream_t stream)
{
    for (int k = 0; k < K_NUM; k++)
        launch_kernel((KernelId)k, jt, ps, q, pp, shape, stream);
}

template <bool kOne>
static void launch_one(KernelId k, const JobTable &jt, const PathState &ps, const Queues &q, int pp,
                       const LaunchShape &shape, const JobView &one, cudaStream_t stream);

void launch_kernel(KernelId k, const JobTable &jt, const PathState &ps, const Queues &q, int pp,
                   const LaunchShape &shape, cudaStream_t stream)
{
    if (jt.only)
        launch_one<true>(k, jt, ps, q, pp, shape, *jt.only, stream);
    else
        launch_one<false>(k, jt, ps, q, pp, shape, JobView{}, stream);
}

template <bool kOne>
static void launch_one(KernelId k, const JobTable &jt, const PathState &ps, const Queues &q, int pp,
                       const LaunchShape &shape, const JobView &one, cudaStream_t stream)
{
    // By default: k_shade's 128 registers let two blocks of 256 share an SM, and
    // two also serve k_regen best, whose accesses get in each other's way beyond
    // that (1080p x 32 medium scene, four and two per SM: shading 47.7 and 46.9
    // ms, regeneration 14.3 and 13.6 ms). With all limits 256 x 256 previews,
    // 131,072 slots, went from 2.63 to 2.37 ms on the device.
    auto blocks = [&](int grid, int per_sm, uint32_t per_block) { return launch_blocks(shape, grid, per_sm, per_block); };
    const uint32_t block = (uint32_t)shape.block;
    switch (k) {
    case K_REGEN:
        k_regen<kOne><<<blocks(shape.grid, 2, block), shape.block, 0, stream>>>(jt, ps, q, pp, one);
        break;
    case K_TRACE:
        // five blocks of k_trace fit an SM where the other kernels' shape counts
        // four; two per SM stay even for few slots, whose rays are spread thin
        k_trace<kOne><<<blocks(shape.grid + shape.grid / 4, 8, std::min(block, shape.slots / (2u * shape.num_sms) + 1u)),
                  shape.block, kTlasCacheBytes, stream>>>(jt, ps, q, pp, one);
        break;
    case K_PARTITION:
        k_partition<<<blocks(shape.grid, 8, 4 * block), shape.block, 0, stream>>>(ps, q, pp);
        break;
    case K_WALK:
        k_walk<<<shape.grid, shape.block, kTlasCacheBytes, stream>>>(jt, ps, q);
        break;
    case K_SHADE:
#if VVPT_SHADE_SPLIT
        k_shade<0, kOne><<<shape.grid, shape.block, kTlasCacheBytes, stream>>>(jt, ps, q, pp, one);
        k_shade<1, kOne><<<shape.grid, shape.block, kTlasCacheBytes, stream>>>(jt, ps, q, pp, one);
        k_shade<2, kOne><<<shape.grid, shape.block, kTlasCacheBytes, stream>>>(jt, ps, q, pp, one);
#else
        k_shade<3, kOne><<<blocks(shape.grid, VVPT_SHADE_MIN_BLOCKS, block), shape.block, kTlasCacheBytes, stream>>>(jt, ps, q, pp, one);
#endif
        break;
    default:
        break;
    }
}

void launch_reduce(const RenderParams &hp, const BatchResults &br, float4 *radiance, float4 *albedo, float4 *normal,
                   float4 *radiance_m2, cudaStream_t stream)
{
    uint32_t npix = hp.width * hp.height;
    int grid = (int)std::min<uint32_t>((npix + 255) / 256, 65535u);
    k_reduce<<<grid, 256, 0, stream>>>(hp, br, radiance, albedo, normal, radiance_m2);
}

void launch_trace_closest(const SceneView &s, const float4 *rays, uint32_t n, vvpt_hit *hits, uint32_t *status,
                          int num_sms, cudaStream_t stream)
{
    const uint32_t full = (uint32_t)num_sms * VVPT_TRACE_MIN_BLOCKS;
    if (n > full * 256u)
        k_trace_closest_refill<<<full, 256, kTlasCacheBytes, stream>>>(s, rays, n, hits, status);
    else
        k_trace_closest<<<std::max((n + 255u) / 256u, 1u), 256, kTlasCacheBytes, stream>>>(s, rays, n, hits, status);
}

}  // namespace vvpt
