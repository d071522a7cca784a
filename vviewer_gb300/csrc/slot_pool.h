// Sizes of the path-slot pools (host code, no CUDA calls).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "wavefront.cuh"

namespace vvpt {

constexpr size_t aligned256(size_t b) { return (b + 255) & ~size_t(255); }

constexpr size_t path_state_bytes(size_t slots) { return slots * sizeof(PathRecord); }

// 11 queues and the counters
constexpr size_t queue_bytes(size_t slots)
{
    return 11 * aligned256(slots * sizeof(uint32_t)) + aligned256(C_COUNT * sizeof(uint32_t));
}

// The idle list of a job table.
constexpr size_t idle_bytes(size_t slots) { return aligned256(slots * sizeof(uint32_t)); }

// Device memory that callers account for (the job engine's budget, the fixed
// scratch of vvpt_render_noalloc) is granted by the size of a path's members,
// 252 bytes: 14 arrays of 16 bytes a slot and 7 of 4. A record takes 256, so one
// slot in 64 stays unused there.
constexpr size_t path_member_bytes(size_t slots)
{
    return 14 * aligned256(slots * 16) + 7 * aligned256(slots * 4);
}
constexpr uint32_t slots_within_members(uint32_t slots)
{
    return (uint32_t)std::min<size_t>(slots, path_member_bytes(slots) / sizeof(PathRecord));
}

}  // namespace vvpt
