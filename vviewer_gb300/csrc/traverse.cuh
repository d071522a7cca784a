// Closest-hit traversal of the two-level BVH (instance TLAS over per-mesh BLAS)
// with a watertight ray/triangle test.
//
// Semantics replaced: traceRayEXT against a TLAS whose instances have culling
// disabled (src/lib/vengine/vulkan/VulkanScene.cpp:375) and an any-hit shader
// that accepts every candidate (shaders/pt/rayPrimary.rahit.glsl:32-71), i.e.
// plain closest hit over [tmin, tmax]. Ties in t are broken by the smallest
// (instance slot, primitive index) so the result does not depend on BVH
// layout; the CPU oracle applies the same rule.
//
// The triangle test is the watertight algorithm of Woop, Benthin and Wald,
// "Watertight Ray/Triangle Intersection", JCGT 2(1), 2013, written with
// explicitly rounded operations (no FMA contraction) so that it gives the same
// bits as a plain IEEE float evaluation on the host.
#pragma once
#include "scene_gpu.h"
#include "vmath.cuh"

namespace vvpt {

// Traversal step counter hook (node visits, triangle tests, instance
// entries) for host builds that measure BVH quality; empty otherwise.
#ifndef VVPT_TRAVERSAL_STAT
#define VVPT_TRAVERSAL_STAT(kind)
#endif

constexpr uint32_t kNoHit = 0xFFFFFFFFu;
// device status word bits
constexpr uint32_t kErrStackOverflow = 1u;
constexpr uint32_t kErrLoopCap = 2u;

struct Hit {
    float t, u, v;
    uint32_t inst, prim;
};

// 1 / x, correctly rounded (the division by another name).
__device__ __forceinline__ float rcp_rn(float x)
{
#ifdef __CUDA_ARCH__
    return __frcp_rn(x);
#else
    return __fdiv_rn(1.0f, x);
#endif
}

// One traversal level's ray: the negated origin (x + (-o) is x - o exactly),
// the inverse direction and the watertight test's shear. kz is the axis of the
// largest direction component and the other two follow it cyclically. The
// published test swaps those two when that component is negative, to keep the
// winding; the swap negates U, V, W, the determinant and T exactly, which
// leaves t, u, v and every decision as they are, so it is left out.
struct LevelRay {
    float3 norg, invd;
    float Sx, Sy, Sz;
    int kz;
};

__device__ __forceinline__ float3 safe_inv(const float3 &d) { return f3(rcp_rn(d.x), rcp_rn(d.y), rcp_rn(d.z)); }

// component kz + 1, kz + 2 or kz of (x, y, z)
__device__ __forceinline__ float axis1(float x, float y, float z, int kz) { return kz == 0 ? y : (kz == 1 ? z : x); }
__device__ __forceinline__ float axis2(float x, float y, float z, int kz) { return kz == 0 ? z : (kz == 1 ? x : y); }
__device__ __forceinline__ float axis0(float x, float y, float z, int kz) { return kz == 0 ? x : (kz == 1 ? y : z); }

__device__ __forceinline__ void level_shear(LevelRay &r, const float3 &d)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    r.kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    const float dz = axis0(d.x, d.y, d.z, r.kz);
    r.Sx = __fdiv_rn(axis1(d.x, d.y, d.z, r.kz), dz);
    r.Sy = __fdiv_rn(axis2(d.x, d.y, d.z, r.kz), dz);
    r.Sz = axis0(r.invd.x, r.invd.y, r.invd.z, r.kz);
}

// Returns true and writes t/u/v when the triangle is hit with t in
// [tmin, best_t]; u, v are the barycentric weights of v1 and v2.
__device__ __forceinline__ bool wt_intersect(const LevelRay &r, const float4 &p0, const float4 &p1, const float4 &p2,
                                             float tmin, float best_t, float &t_out, float &u_out, float &v_out)
{
    const float Ax0 = __fadd_rn(p0.x, r.norg.x), Ay0 = __fadd_rn(p0.y, r.norg.y), Az0 = __fadd_rn(p0.z, r.norg.z);
    const float Bx0 = __fadd_rn(p1.x, r.norg.x), By0 = __fadd_rn(p1.y, r.norg.y), Bz0 = __fadd_rn(p1.z, r.norg.z);
    const float Cx0 = __fadd_rn(p2.x, r.norg.x), Cy0 = __fadd_rn(p2.y, r.norg.y), Cz0 = __fadd_rn(p2.z, r.norg.z);
    const float Az = axis0(Ax0, Ay0, Az0, r.kz), Bz = axis0(Bx0, By0, Bz0, r.kz), Cz = axis0(Cx0, Cy0, Cz0, r.kz);
    const float ax = __fsub_rn(axis1(Ax0, Ay0, Az0, r.kz), __fmul_rn(r.Sx, Az));
    const float ay = __fsub_rn(axis2(Ax0, Ay0, Az0, r.kz), __fmul_rn(r.Sy, Az));
    const float bx = __fsub_rn(axis1(Bx0, By0, Bz0, r.kz), __fmul_rn(r.Sx, Bz));
    const float by = __fsub_rn(axis2(Bx0, By0, Bz0, r.kz), __fmul_rn(r.Sy, Bz));
    const float cx = __fsub_rn(axis1(Cx0, Cy0, Cz0, r.kz), __fmul_rn(r.Sx, Cz));
    const float cy = __fsub_rn(axis2(Cx0, Cy0, Cz0, r.kz), __fmul_rn(r.Sy, Cz));
    float U = __fsub_rn(__fmul_rn(cx, by), __fmul_rn(cy, bx));
    float V = __fsub_rn(__fmul_rn(ax, cy), __fmul_rn(ay, cx));
    float W = __fsub_rn(__fmul_rn(bx, ay), __fmul_rn(by, ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        // edge case: redo the 2D edge tests in double precision
        double cxby = __dmul_rn((double)cx, (double)by), cybx = __dmul_rn((double)cy, (double)bx);
        U = (float)__dsub_rn(cxby, cybx);
        double axcy = __dmul_rn((double)ax, (double)cy), aycx = __dmul_rn((double)ay, (double)cx);
        V = (float)__dsub_rn(axcy, aycx);
        double bxay = __dmul_rn((double)bx, (double)ay), byax = __dmul_rn((double)by, (double)ax);
        W = (float)__dsub_rn(bxay, byax);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f))
        return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f)
        return false;
    const float az = __fmul_rn(r.Sz, Az), bz = __fmul_rn(r.Sz, Bz), cz = __fmul_rn(r.Sz, Cz);
    const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, az), __fmul_rn(V, bz)), __fmul_rn(W, cz));
    const float rcp = rcp_rn(det);
    const float t = __fmul_rn(T, rcp);
    if (!(t >= tmin) || !(t <= best_t))
        return false;
    t_out = t;
    u_out = __fmul_rn(V, rcp);
    v_out = __fmul_rn(W, rcp);
    return true;
}

// Strictly after `a` in (t, instance, primitive) order; a.inst == kNoHit
// means no constraint. Used to walk any-hit candidates nearest first.
__device__ __forceinline__ bool is_after(float t, uint32_t inst, uint32_t prim, const Hit &a)
{
    if (a.inst == kNoHit)
        return true;
    if (t != a.t)
        return t > a.t;
    if (inst != a.inst)
        return inst > a.inst;
    return prim > a.prim;
}

__device__ __forceinline__ bool better(float t, uint32_t inst, uint32_t prim, const Hit &h)
{
    if (t != h.t)
        return t < h.t;
    if (inst != h.inst)
        return inst < h.inst;
    return prim < h.prim;
}

// Two floats per instruction (sm_100 and later), each rounded on its own:
// (a - o) * invd with the origin negated.
__device__ __forceinline__ void slab2(float a0, float a1, float no0, float no1, float i0, float i1, float &t0, float &t1)
{
#ifdef __CUDA_ARCH__
    asm("{ .reg .b64 a, b;\n\t"
        "mov.b64 a, {%2, %3};\n\t"
        "mov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 a, a, b;\n\t"
        "mov.b64 b, {%6, %7};\n\t"
        "mul.rn.f32x2 a, a, b;\n\t"
        "mov.b64 {%0, %1}, a; }"
        : "=f"(t0), "=f"(t1)
        : "f"(a0), "f"(a1), "f"(no0), "f"(no1), "f"(i0), "f"(i1));
#else
    t0 = __fmul_rn(__fadd_rn(a0, no0), i0);
    t1 = __fmul_rn(__fadd_rn(a1, no1), i1);
#endif
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
#else
    return fminf(fminf(a, b), c);
#endif
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}

// Conservative slab test (Pharr, Jakob, Humphreys, PBRT 3rd ed. sec. 3.9.2:
// (lo - o) * invd with tfar scaled by 1 + 2*gamma(3)) of both children of a
// node: whether each is touched within [tmin, tmax], and its entry distance.
__device__ __forceinline__ void box2(const BVHNode &n, const LevelRay &r, float tmin, float tmax, bool &hl, bool &hr,
                                     float &tl, float &tr)
{
    const float kScale = 1.0f + 2.0f * 3.5762793e-07f; // 1 + 2*gamma(3), gamma(3) = 3u/(1-3u), u = 2^-24
    float lx0, lx1, ly0, ly1, lz0, lz1, rx0, rx1, ry0, ry1, rz0, rz1;
    slab2(n.lxy.x, n.lxy.y, r.norg.x, r.norg.y, r.invd.x, r.invd.y, lx0, ly0);
    slab2(n.lxy.z, n.lxy.w, r.norg.x, r.norg.y, r.invd.x, r.invd.y, lx1, ly1);
    slab2(n.rxy.x, n.rxy.y, r.norg.x, r.norg.y, r.invd.x, r.invd.y, rx0, ry0);
    slab2(n.rxy.z, n.rxy.w, r.norg.x, r.norg.y, r.invd.x, r.invd.y, rx1, ry1);
    slab2(n.lrz.x, n.lrz.y, r.norg.z, r.norg.z, r.invd.z, r.invd.z, lz0, lz1);
    slab2(n.lrz.z, n.lrz.w, r.norg.z, r.norg.z, r.invd.z, r.invd.z, rz0, rz1);
    tl = fmaxf(max3(fminf(lx0, lx1), fminf(ly0, ly1), fminf(lz0, lz1)), tmin);
    tr = fmaxf(max3(fminf(rx0, rx1), fminf(ry0, ry1), fminf(rz0, rz1)), tmin);
    const float lfar = fminf(min3(fmaxf(lx0, lx1), fmaxf(ly0, ly1), fmaxf(lz0, lz1)), tmax) * kScale;
    const float rfar = fminf(min3(fmaxf(rx0, rx1), fmaxf(ry0, ry1), fmaxf(rz0, rz1)), tmax) * kScale;
    hl = tl <= lfar && n.c.x >= 0;
    hr = tr <= rfar && n.c.y >= 0;
}

// Culling bounds with slack. A node is skipped when its entry distance lies
// beyond the current best hit. The slab distances and the triangle test's t
// carry independent rounding errors, so for a triangle on a node's face
// (coplanar geometry, axis-aligned walls) the computed entry can exceed the
// computed hit t. Two margins keep such nodes (and equal-t ties, which the
// (instance, primitive) order resolves) in the search: 1e-5 relative to t, and
// an absolute one for hits close to the ray origin, where the triangle's t is
// a difference of coordinates far larger than t itself and its error is about
// machine epsilon times those coordinates over |d| (cull_slack).
__device__ __forceinline__ float cull_far(float best_t, float slack)
{
    return best_t * (1.0f + 1e-5f) + slack + 1e-30f;
}
__device__ __forceinline__ float cull_near(float tmin, float slack) { return tmin - fabsf(tmin) * 1e-5f - slack; }
// Absolute culling margin of one ray: 1e-5 (about 160 ulps) times the largest
// object-space coordinate magnitude a triangle test of this scene can see,
// bounded per instance on the host (SceneView::cull_o, cull_r), over |d|.
__device__ __forceinline__ float cull_slack(const SceneView &s, const float3 &o, const float3 &d)
{
    const float om = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
    const float dm = fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
    return dm > 0.0f ? 1e-5f * (s.cull_o * om + s.cull_r) / dm : 0.0f;
}

// Loads of BVH nodes and triangles. With VVPT_SCENE_L2_KEEP = 1 (a build
// option) they carry an L2 evict-last policy, so that the scene's lines,
// re-read by every traversal kernel, outlive the path state and queues that
// stream through L2. Measured on the 1080p medium scene: no gain (137.3
// against 140.3 M paths/s without it, within run-to-run spread), so off.
#ifndef VVPT_SCENE_L2_KEEP
#define VVPT_SCENE_L2_KEEP 0
#endif
#if defined(__CUDA_ARCH__) && VVPT_SCENE_L2_KEEP
__device__ __forceinline__ uint64_t scene_l2_policy()
{
    uint64_t pol;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ float4 ldg_scene(const float4 *p)
{
    float4 v;
    asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p), "l"(scene_l2_policy()));
    return v;
}
#else
__device__ __forceinline__ float4 ldg_scene(const float4 *p) { return __ldg(p); }
#endif

__device__ __forceinline__ BVHNode load_node(const BVHNode *nodes, int idx)
{
    const float4 *p = reinterpret_cast<const float4 *>(nodes + idx);
    BVHNode n;
    n.lxy = ldg_scene(p + 0);
    n.rxy = ldg_scene(p + 1);
    n.lrz = ldg_scene(p + 2);
    float4 c = ldg_scene(p + 3);
    n.c = make_int4(__float_as_int(c.x), __float_as_int(c.y), __float_as_int(c.z), __float_as_int(c.w));
    return n;
}

// Object-space ray of an instance, with explicitly rounded arithmetic so the
// host oracle reproduces it exactly: ((m0*x + m1*y) + m2*z) + m3.
__device__ __forceinline__ float3 wt_xform_point(const float4 *rows, const float3 &p)
{
    float3 r;
    r.x = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(rows[0].x, p.x), __fmul_rn(rows[0].y, p.y)), __fmul_rn(rows[0].z, p.z)), rows[0].w);
    r.y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(rows[1].x, p.x), __fmul_rn(rows[1].y, p.y)), __fmul_rn(rows[1].z, p.z)), rows[1].w);
    r.z = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(rows[2].x, p.x), __fmul_rn(rows[2].y, p.y)), __fmul_rn(rows[2].z, p.z)), rows[2].w);
    return r;
}
__device__ __forceinline__ float3 wt_xform_vector(const float4 *rows, const float3 &v)
{
    float3 r;
    r.x = __fadd_rn(__fadd_rn(__fmul_rn(rows[0].x, v.x), __fmul_rn(rows[0].y, v.y)), __fmul_rn(rows[0].z, v.z));
    r.y = __fadd_rn(__fadd_rn(__fmul_rn(rows[1].x, v.x), __fmul_rn(rows[1].y, v.y)), __fmul_rn(rows[1].z, v.z));
    r.z = __fadd_rn(__fadd_rn(__fmul_rn(rows[2].x, v.x), __fmul_rn(rows[2].y, v.y)), __fmul_rn(rows[2].z, v.z));
    return r;
}

#if VVPT_BLAS_WIDE
// Byte k of w as an exact float: 0x4B0000bb is the float 2^23 + bb.
__device__ __forceinline__ float byte_as_float(uint32_t w, int k)
{
    return __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (uint32_t)k)), 8388608.0f);
}

// Ray against the 8 child boxes of a wide node (five 128-bit words `w`).
// Per axis the node gives the slab distance of a plane q as one multiply-add,
// q * A + B with A = scale * invd and B = (p - o) * invd, near and far planes
// chosen by the sign of the inverse direction. That form rounds relative to
// |B| + 255 |A| rather than to the distance itself (the two terms cancel near
// the plane), so each axis carries its own margin, 8 ulps of |B| + 255 |A|
// (several times the worst-case error of the four roundings), folded into B:
// near distances move down and far ones up, and no child the ray touches is
// missed (a zero direction component gives infinities or NaN there, and NaN
// leaves that axis unconstrained). Outputs: the internal-child hits at bit
// (slot ^ oct), the node's imask and child_base, and the hit leaf children's
// triangles as a mask over tri_base + 0..31.
__device__ __forceinline__ void wide_visit(const float4 (&w)[5], const float3 &norg, const float3 &invd, uint32_t oct,
                                           float tmin, float tmax, uint32_t &node_bits, uint32_t &imask,
                                           uint32_t &child_base, uint32_t &tri_base, uint32_t &tri_bits)
{
    const uint32_t eim = __float_as_uint(w[0].w);
    const float ax = __fmul_rn(__uint_as_float((eim & 0xffu) << 23), invd.x);
    const float ay = __fmul_rn(__uint_as_float(((eim >> 8) & 0xffu) << 23), invd.y);
    const float az = __fmul_rn(__uint_as_float(((eim >> 16) & 0xffu) << 23), invd.z);
    const float bx = __fmul_rn(__fadd_rn(w[0].x, norg.x), invd.x);
    const float by = __fmul_rn(__fadd_rn(w[0].y, norg.y), invd.y);
    const float bz = __fmul_rn(__fadd_rn(w[0].z, norg.z), invd.z);
    const float kUlps = 8.0f * 5.9604645e-08f; // 8 x 2^-24
    const float mx = __fmul_rn(kUlps, __fmaf_rn(255.0f, fabsf(ax), fabsf(bx)));
    const float my = __fmul_rn(kUlps, __fmaf_rn(255.0f, fabsf(ay), fabsf(by)));
    const float mz = __fmul_rn(kUlps, __fmaf_rn(255.0f, fabsf(az), fabsf(bz)));
    const float bnx = __fsub_rn(bx, mx), bfx = __fadd_rn(bx, mx);
    const float bny = __fsub_rn(by, my), bfy = __fadd_rn(by, my);
    const float bnz = __fsub_rn(bz, mz), bfz = __fadd_rn(bz, mz);
    imask = eim >> 24;
    child_base = __float_as_uint(w[1].x);
    tri_base = __float_as_uint(w[1].y);
    const uint32_t meta[2] = {__float_as_uint(w[1].z), __float_as_uint(w[1].w)};
    const bool nx = (oct & 1u) != 0, ny = (oct & 2u) != 0, nz = (oct & 4u) != 0;
    // near / far plane words per axis: lo (w2.xy, w2.zw, w3.xy), hi (w3.zw, w4.xy, w4.zw)
    const uint32_t nxw[2] = {__float_as_uint(nx ? w[3].z : w[2].x), __float_as_uint(nx ? w[3].w : w[2].y)};
    const uint32_t fxw[2] = {__float_as_uint(nx ? w[2].x : w[3].z), __float_as_uint(nx ? w[2].y : w[3].w)};
    const uint32_t nyw[2] = {__float_as_uint(ny ? w[4].x : w[2].z), __float_as_uint(ny ? w[4].y : w[2].w)};
    const uint32_t fyw[2] = {__float_as_uint(ny ? w[2].z : w[4].x), __float_as_uint(ny ? w[2].w : w[4].y)};
    const uint32_t nzw[2] = {__float_as_uint(nz ? w[4].z : w[3].x), __float_as_uint(nz ? w[4].w : w[3].y)};
    const uint32_t fzw[2] = {__float_as_uint(nz ? w[3].x : w[4].z), __float_as_uint(nz ? w[3].y : w[4].w)};
    node_bits = 0;
    tri_bits = 0;
#pragma unroll 2
    for (int i = 0; i < 8; i++) {
        const int h = i >> 2, k = i & 3;
        const float tnx = __fmaf_rn(byte_as_float(nxw[h], k), ax, bnx);
        const float tfx = __fmaf_rn(byte_as_float(fxw[h], k), ax, bfx);
        const float tny = __fmaf_rn(byte_as_float(nyw[h], k), ay, bny);
        const float tfy = __fmaf_rn(byte_as_float(fyw[h], k), ay, bfy);
        const float tnz = __fmaf_rn(byte_as_float(nzw[h], k), az, bnz);
        const float tfz = __fmaf_rn(byte_as_float(fzw[h], k), az, bfz);
        const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, tmin));
        const float tf = fminf(fminf(tfx, tfy), fminf(tfz, tmax));
        if (tn <= tf) {
            const uint32_t m = (meta[h] >> (8 * k)) & 0xffu;
            if ((imask >> i) & 1u)
                node_bits |= 1u << (i ^ (int)oct);
            else if (m)
                tri_bits |= ((1u << (m >> 5)) - 1u) << (m & 31u);
        }
    }
}

__device__ __forceinline__ void load_wide(const WideNode *nodes, uint32_t idx, float4 (&w)[5])
{
    const float4 *p = reinterpret_cast<const float4 *>(nodes + idx);
#pragma unroll
    for (int k = 0; k < 5; k++)
        w[k] = __ldg(p + k);
}
#endif

// Top of the TLAS staged in shared memory: a traversal kernel fills it at its
// start with the first kTlasCacheNodes nodes of one live scene (the scene of
// its block's first queue entry; launched with kTlasCacheBytes of dynamic
// shared memory), and trace_after reads TLAS nodes of that scene from it.
// Kernels that do not fill it clear it (tlas_cache_none).
constexpr int kTlasCacheNodes = 128;
constexpr int kTlasCacheBytes = kTlasCacheNodes * (int)sizeof(BVHNode);
extern __shared__ __align__(16) float4 vvpt_tlas_cache[];
__shared__ const BVHNode *vvpt_tlas_cache_src;
__shared__ int vvpt_tlas_cache_count;

#ifdef __CUDACC__
__device__ __forceinline__ void tlas_cache_fill(const SceneView &s)
{
    const BVHNode *src = s.nodes + s.tlas_root;
    const int cnt = min((int)s.tlas_count, kTlasCacheNodes);
    const float4 *f = reinterpret_cast<const float4 *>(src);
    for (int i = threadIdx.x; i < 4 * cnt; i += blockDim.x)
        vvpt_tlas_cache[i] = __ldg(f + i);
    if (threadIdx.x == 0) {
        vvpt_tlas_cache_src = src;
        vvpt_tlas_cache_count = cnt;
    }
    __syncthreads();
}

__device__ __forceinline__ void tlas_cache_none()
{
    if (threadIdx.x == 0) {
        vvpt_tlas_cache_src = nullptr;
        vvpt_tlas_cache_count = 0;
    }
    __syncthreads();
}
#endif

__device__ __forceinline__ BVHNode load_node_cached(int idx)
{
    const float4 *p = vvpt_tlas_cache + 4 * idx;
    BVHNode n;
    n.lxy = p[0];
    n.rxy = p[1];
    n.lrz = p[2];
    const float4 c = p[3];
    n.c = make_int4(__float_as_int(c.x), __float_as_int(c.y), __float_as_int(c.z), __float_as_int(c.w));
    return n;
}

// Closest hit over all TLAS instances among candidates strictly after
// `after`, as one flat loop over a single stack. Every loop step is one of: a
// triangle test, or a node visit (both children's boxes) with the stack
// transitions before it (enter an instance: transform the ray into its object
// space; leave it: back to the world-space ray). Keeping the two levels in one
// loop keeps a warp's lanes in step: a lane inside an instance never holds
// lanes that are still in the TLAS, as nested per-level loops would. The
// nearer child goes first, at both levels, and a stack entry carries its entry
// distance, so that what a hit found meanwhile has put out of reach is dropped
// when it is popped (the test a visit of its parent would make now) instead of
// being loaded and tested. The loop's state lives in a TraceState and one step
// is trace_step, so that a kernel can also run the steps of several rays on
// one lane, one after the other (trace_after is the one-ray loop). `err`
// receives status bits.
//
// Bound by instruction issue under divergence, so the form is about the
// instructions and steps of a ray: boxes two floats per instruction with
// three-way minima, no step that only pops, reciprocals instead of divisions,
// the shear only where triangles can follow. Host step counts against far
// child and popped entries always visited: camera rays into the medium room
// 22.0 -> 11.9 steps, into the open sky scene 52.4 -> 46.6, diffuse bounces
// there 45.0 -> 43.4. Trace launches of the 1080p medium scene (32 spp):
// 211 -> 167 ms, of the sky scene 54.5 -> 44.2 ms.
//
// References, the kind in the two top bits: an inner node (index from the
// level's first node), a triangle run of a leaf (first triangle; TriVerts::v2.w
// marks the last), an instance run of a TLAS leaf (index into tlas_order, whose
// top bit marks the last), the return from an instance; kRefDone ends the ray.
constexpr uint32_t kRefLeaf = 1u << 30, kRefInst = 2u << 30, kRefReturn = 3u << 30, kRefDone = 0xFFFFFFFFu;
constexpr uint32_t kRefIndex = kMaxRefIndex;
#if VVPT_BLAS_WIDE
constexpr uint32_t kRefWide = 1u << 30; // wide children still to visit (its BLAS has no leaf references)
#endif

// What a node visit does not read: the world-space ray, the best hit so far
// and the current instance. The refill loop keeps it in shared memory, one
// array per member, and its registers for the visit.
struct TraceCold {
    float4 &o_slack; // origin, absolute culling margin
    float4 &d_tmin;  // direction, tmin
    float4 &best;    // best hit so far: t, u, v, primitive (bits)
    uint2 &ids;      // its instance, the instance whose BLAS is traversed
};

struct TraceState {
    float box_tmin;
    float far_t;         // culling distance of the best hit so far
    LevelRay lr;         // the level's ray; in the TLAS its shear is not set and kz is kInTlas
    uint32_t node_base;
    uint32_t tri_base;   // in the TLAS: nodes below this index come from shared memory
    uint32_t cur;        // next reference
    int sp, floor;       // stack entries; those of the level above
#if VVPT_BLAS_WIDE
    // BLAS level: the group of wide children still to visit (hits at bit
    // slot ^ oct, imask, first child) and the triangles still to test (mask
    // over t_base + 0..31); oct = sign bits of the object-space direction
    uint32_t w_base, w_bits, w_imask, t_base, t_bits, oct;
#endif
};
constexpr int kInTlas = 3;
// The traversal stack (reference, entry distance), kept apart from the scalar
// state so that the scalars stay in registers.
typedef int2 TraceStack[kTraversalStack];

__device__ __forceinline__ Hit trace_best(const TraceCold &c)
{
    Hit h;
    h.t = c.best.x;
    h.u = c.best.y;
    h.v = c.best.z;
    h.prim = __float_as_uint(c.best.w);
    h.inst = c.ids.x;
    return h;
}

// The world-space ray at the TLAS.
__device__ __forceinline__ void trace_enter_tlas(TraceState &st, const SceneView &s, const float3 &o, const float3 &d)
{
    st.lr.norg = -o;
    st.lr.invd = safe_inv(d);
    st.lr.kz = kInTlas;
    st.node_base = s.tlas_root;
    st.tri_base = vvpt_tlas_cache_src == s.nodes + s.tlas_root ? (uint32_t)vvpt_tlas_cache_count : 0u;
    st.floor = 0;
}

__device__ __forceinline__ void trace_begin(TraceState &st, const TraceCold &c, const SceneView &s, const float3 &o,
                                            const float3 &d, float tmin, float tmax, const Hit &after)
{
    const float slack = cull_slack(s, o, d);
    c.o_slack = make_float4(o.x, o.y, o.z, slack);
    c.d_tmin = make_float4(d.x, d.y, d.z, tmin);
    c.best = make_float4(tmax, 0.0f, 0.0f, __uint_as_float(kNoHit));
    c.ids = make_uint2(kNoHit, kNoHit);
    st.far_t = cull_far(tmax, slack);
    st.box_tmin = cull_near(after.inst == kNoHit ? tmin : fmaxf(tmin, after.t), slack);
    st.lr.Sx = st.lr.Sy = st.lr.Sz = 0.0f;
    trace_enter_tlas(st, s, o, d);
    st.cur = 0;
#if VVPT_BLAS_WIDE
    st.w_base = st.w_bits = st.w_imask = st.t_base = st.t_bits = st.oct = 0;
#endif
    st.sp = 0;
}

__device__ __forceinline__ void trace_push(TraceState &st, TraceStack &stack, uint32_t ref, float t, uint32_t &err)
{
    if (st.sp < kTraversalStack)
        stack[st.sp++] = make_int2((int)ref, __float_as_int(t));
    else
        err |= kErrStackOverflow;
}

// The next reference of the level, of those still in reach; with none left,
// the return to the TLAS or the end of the ray.
__device__ __forceinline__ uint32_t trace_pop(TraceState &st, const TraceStack &stack)
{
    while (st.sp > st.floor) {
        const int2 e = stack[--st.sp];
#if VVPT_BLAS_WIDE
        if (((uint32_t)e.x >> 30) == 1u) { // a group's bits in place of a distance
            st.w_base = (uint32_t)e.x & kRefIndex;
            st.w_bits = ((uint32_t)e.y >> 8) & 0xffu;
            st.w_imask = (uint32_t)e.y & 0xffu;
            return kRefWide;
        }
#endif
        if (__int_as_float(e.y) <= st.far_t)
            return (uint32_t)e.x;
    }
    return st.lr.kz != kInTlas ? kRefReturn : kRefDone;
}

// Tests one triangle of the current BLAS against the ray and keeps it when it
// is the best candidate after `after`; whether it is its leaf's last.
__device__ __forceinline__ bool trace_triangle(TraceState &st, const TraceCold &c, const SceneView &s, uint32_t local,
                                               const Hit &after)
{
    const float4 *tp = reinterpret_cast<const float4 *>(s.tris + st.tri_base + local);
    const float4 p0 = ldg_scene(tp), p1 = ldg_scene(tp + 1), p2 = ldg_scene(tp + 2);
    float t, u, v;
    if (wt_intersect(st.lr, p0, p1, p2, c.d_tmin.w, c.best.x, t, u, v)) {
        const uint32_t prim = __float_as_uint(p0.w);
        const uint32_t tag = __float_as_uint(p1.w);
        const uint32_t hinst = tag ? tag - 1u : c.ids.y; // baked triangles name their instance
        if (better(t, hinst, prim, trace_best(c)) && is_after(t, hinst, prim, after)) {
            c.best = make_float4(t, u, v, p0.w);
            c.ids.x = hinst;
            st.far_t = cull_far(t, c.o_slack.w);
        }
    }
    return __float_as_uint(p2.w) != 0u;
}

// The kind of a ray's next step: a node visit, a triangle test, or a
// transition between the levels (enter or leave an instance).
constexpr int kStepNode = 0, kStepTriangle = 1, kStepLevel = 2;
__device__ __forceinline__ int trace_kind(const TraceState &st)
{
#if VVPT_BLAS_WIDE
    if (st.t_bits)
        return kStepTriangle;
    if (st.cur == kRefWide)
        return kStepNode;
#endif
    const uint32_t k = st.cur >> 30;
    return k < 2u ? (int)k : kStepLevel;
}

__device__ __forceinline__ void trace_step_triangle(TraceState &st, const TraceCold &c, TraceStack &stack,
                                                    const SceneView &s, const Hit &after)
{
    VVPT_TRAVERSAL_STAT(1);
#if VVPT_BLAS_WIDE
    const int b = __ffs((int)st.t_bits) - 1;
    st.t_bits &= st.t_bits - 1u;
    trace_triangle(st, c, s, st.t_base + (uint32_t)b, after);
    if (!st.t_bits && !st.w_bits)
        st.cur = trace_pop(st, stack);
#else
    st.cur = trace_triangle(st, c, s, st.cur & kRefIndex, after) ? trace_pop(st, stack) : st.cur + 1u;
#endif
}

__device__ __forceinline__ void trace_step_level(TraceState &st, const TraceCold &c, TraceStack &stack,
                                                 const SceneView &s, uint32_t &err)
{
    if (st.cur == kRefReturn) {
        trace_enter_tlas(st, s, f3(c.o_slack), f3(c.d_tmin));
        st.cur = trace_pop(st, stack);
    }
    if ((st.cur >> 30) == 2u) {
        VVPT_TRAVERSAL_STAT(2);
        const uint32_t at = st.cur & kRefIndex;
        const uint32_t id = __ldg(s.tlas_order + at);
        if (!(id >> 31))
            trace_push(st, stack, kRefInst | (at + 1u), st.box_tmin, err);
        c.ids.y = id & 0x7FFFFFFFu;
        const DevInstance &inst = s.instances[id & 0x7FFFFFFFu];
        const float4 rows[3] = {inst.w2o[0], inst.w2o[1], inst.w2o[2]};
        const float3 cd = wt_xform_vector(rows, f3(c.d_tmin));
        st.lr.norg = -wt_xform_point(rows, f3(c.o_slack));
        st.lr.invd = safe_inv(cd);
        level_shear(st.lr, cd);
        st.node_base = inst.node_offset;
        st.tri_base = inst.tri_offset;
        st.floor = st.sp;
#if VVPT_BLAS_WIDE
        // the BLAS root as a one-child group
        st.oct = (__float_as_uint(cd.x) >> 31) | ((__float_as_uint(cd.y) >> 31) << 1) |
                 ((__float_as_uint(cd.z) >> 31) << 2);
        st.w_base = 0;
        st.w_imask = 1u;
        st.w_bits = 1u << st.oct;
        st.cur = kRefWide;
#else
        st.cur = 0;
#endif
    }
}

__device__ __forceinline__ void trace_step_node(TraceState &st, TraceStack &stack, const SceneView &s, uint32_t &err)
{
#if VVPT_BLAS_WIDE
    if (st.cur == kRefWide) {
        // nearest remaining child of the group (octant order)
        const int b = __ffs((int)st.w_bits) - 1;
        st.w_bits &= st.w_bits - 1u;
        const uint32_t slot = (uint32_t)b ^ st.oct;
        const uint32_t child = st.w_base + (uint32_t)__popc(st.w_imask & ((1u << slot) - 1u));
        if (st.w_bits)
            trace_push(st, stack, kRefWide | st.w_base, __int_as_float((int)((st.w_bits << 8) | st.w_imask)), err);
        float4 wn[5];
        load_wide(s.wnodes, st.node_base + child, wn);
        wide_visit(wn, st.lr.norg, st.lr.invd, st.oct, st.box_tmin, st.far_t, st.w_bits, st.w_imask, st.w_base,
                   st.t_base, st.t_bits);
        if (!st.t_bits && !st.w_bits)
            st.cur = trace_pop(st, stack);
        return;
    }
#endif
    const bool tlas = st.lr.kz == kInTlas;
    VVPT_TRAVERSAL_STAT(tlas ? 3 : 0);
    const BVHNode n = (tlas && st.cur < st.tri_base) ? load_node_cached((int)st.cur)
                                                        : load_node(s.nodes, (int)(st.node_base + st.cur));
    bool hl, hr;
    float tl, tr;
    box2(n, st.lr, st.box_tmin, st.far_t, hl, hr, tl, tr);
    const uint32_t leaf = tlas ? kRefInst : kRefLeaf;
    const uint32_t lref = (uint32_t)n.c.x | (n.c.z ? leaf : 0u), rref = (uint32_t)n.c.y | (n.c.w ? leaf : 0u);
    if (hl || hr) {
        const bool both = hl && hr, right = both ? tr < tl : hr;
        st.cur = right ? rref : lref;
        if (both)
            trace_push(st, stack, right ? lref : rref, right ? tl : tr, err);
    } else {
        st.cur = trace_pop(st, stack);
    }
}

// One loop step of the one-ray loop, a transition together with the visit
// that follows it; false when the traversal is over (trace_best is the result).
__device__ __forceinline__ bool trace_step(TraceState &st, const TraceCold &c, TraceStack &stack, const SceneView &s,
                                           const Hit &after, uint32_t &err)
{
    if (trace_kind(st) == kStepTriangle) {
        trace_step_triangle(st, c, stack, s, after);
    } else {
        if (trace_kind(st) == kStepLevel)
            trace_step_level(st, c, stack, s, err);
        if (trace_kind(st) == kStepNode)
            trace_step_node(st, stack, s, err);
    }
    return st.cur != kRefDone;
}

__device__ __forceinline__ Hit trace_after(const SceneView &s, const float3 &o, const float3 &d, float tmin, float tmax,
                                           const Hit &after, uint32_t &err)
{
    TraceState st;
    float4 o_slack, d_tmin, best;
    uint2 ids;
    const TraceCold c{o_slack, d_tmin, best, ids};
    TraceStack stack;
    trace_begin(st, c, s, o, d, tmin, tmax, after);
    while (trace_step(st, c, stack, s, after, err)) {
    }
    return trace_best(c);
}

__device__ __forceinline__ Hit no_hit()
{
    Hit h;
    h.t = -1.0f;
    h.u = h.v = 0.0f;
    h.inst = kNoHit;
    h.prim = kNoHit;
    return h;
}

__device__ __forceinline__ Hit trace_closest(const SceneView &s, const float3 &o, const float3 &d, float tmin, float tmax,
                                             uint32_t &err)
{
    return trace_after(s, o, d, tmin, tmax, no_hit(), err);
}

// A BSDF-direction emitter ray adds radiance only at an emissive surface,
// and its candidate walk keeps the direction and moves the origin along the
// line, so it can contribute only if the half-line from `o` along `d` meets
// one of the scene's emissive boxes. The slab interval of each axis is
// widened by 1e-5 of its ends (far above float rounding) and the boxes are
// padded, so a ray that reaches an emitter is never rejected.
__device__ __forceinline__ bool may_reach_emitter(const SceneView &s, const float3 &o, const float3 &d)
{
    const float big = 3.402823466e38f; // NaN and infinities fail |x| <= big
    if (!(fabsf(o.x) <= big && fabsf(o.y) <= big && fabsf(o.z) <= big && fabsf(d.x) <= big && fabsf(d.y) <= big &&
          fabsf(d.z) <= big))
        return true;
    for (uint32_t k = 0; k < s.num_emit_boxes; k++) {
        const float4 lo = __ldg(&s.emit_boxes[2 * k]), hi = __ldg(&s.emit_boxes[2 * k + 1]);
        float t0 = 0.0f, t1 = INFINITY;
        bool out = false;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const float oa = a == 0 ? o.x : (a == 1 ? o.y : o.z);
            const float da = a == 0 ? d.x : (a == 1 ? d.y : d.z);
            const float la = a == 0 ? lo.x : (a == 1 ? lo.y : lo.z);
            const float ha = a == 0 ? hi.x : (a == 1 ? hi.y : hi.z);
            if (da == 0.0f) {
                out |= oa < la || oa > ha;
            } else {
                const float ta = (la - oa) / da, tb = (ha - oa) / da;
                float tn = fminf(ta, tb), tf = fmaxf(ta, tb);
                tn -= 1e-5f * fabsf(tn);
                tf += 1e-5f * fabsf(tf);
                t0 = fmaxf(t0, tn);
                t1 = fminf(t1, tf);
            }
        }
        if (!out && t0 <= t1)
            return true;
    }
    return false;
}

}  // namespace vvpt
