// Test harness: scene packing (vviewer_gb300/csrc/scene_pack.cpp) with a
// builder outside that takes no mesh, against packing without one.
#include <cuda_runtime.h>

#include <cstring>
#include <string>
#include <vector>

#include "bvh_build.h"
#include "scene_pack.h"

using namespace vvpt;

template <class T>
static bool same(const std::vector<T> &a, const std::vector<T> &b)
{
    return a.size() == b.size() && (a.empty() || std::memcmp(a.data(), b.data(), a.size() * sizeof(T)) == 0);
}

extern "C" int host_pack_status(const vvpt_scene_desc *desc, char *msg, int msg_len)
{
    PackedScene packed;
    std::string err;
    const vvpt_status st = pack_scene(desc, packed, err, 2);
    std::strncpy(msg, err.c_str(), msg_len - 1);
    msg[msg_len - 1] = 0;
    return (int)st;
}

// 0: the packed scenes are the same; else the status with `msg`, or -1 where
// they differ. `failure`: what the outside builder reports ("" declines).
extern "C" int host_pack_outside(const vvpt_scene_desc *desc, const char *failure, int *asked, char *msg, int msg_len)
{
    PackedScene plain, packed;
    std::string err;
    if (pack_scene(desc, plain, err, 2) != VVPT_OK)
        return -2;
    OutsideMeshes outside;
    outside.min_triangles = 100;
    outside.tree = [](const std::vector<Box3> &, const BVHBuildOptions &, BVHBuildResult &, std::string &) { return false; };
    outside.build = [&](const std::vector<uint32_t> &meshes, std::vector<MeshPlace> &, std::string &e) {
        *asked = (int)meshes.size();
        e = failure;
        return false;
    };
    const vvpt_status st = pack_scene(desc, packed, err, 2, &outside);
    if (st != VVPT_OK) {
        std::strncpy(msg, err.c_str(), msg_len - 1);
        msg[msg_len - 1] = 0;
        return (int)st;
    }
    return same(plain.nodes, packed.nodes) && same(plain.wnodes, packed.wnodes) && same(plain.tris, packed.tris) &&
                   same(plain.verts, packed.verts) && same(plain.indices, packed.indices) &&
                   same(plain.instances, packed.instances) && same(plain.tlas_order, packed.tlas_order) &&
                   plain.tlas_root == packed.tlas_root
               ? 0
               : -1;
}
