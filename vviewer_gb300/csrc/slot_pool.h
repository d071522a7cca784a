// Path-slot pools: their sizes, and the pool that vvpt_render keeps (host code;
// the CUDA calls come with the Mem parameter).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

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

// A render's pool: records, queues, idle list.
constexpr size_t pool_bytes(size_t slots) { return path_state_bytes(slots) + queue_bytes(slots) + idle_bytes(slots); }

// Path slots of a render whose tuning leaves them open. More slots mean fewer,
// larger launches, and paths that start together: their rays stay neighbours
// on the image for longer, and less of the time goes by waiting for a launch's
// last rays. 2^20 slots (0.3 GB with their queues), 2^22 and 2^24 (5.1 GB):
// 225, 196 and 184 ms on the 1080p x 32 medium scene, 62, 52 and 51 ms on the
// 1919 x 1079 x 16 sky scene. A render has at most one slot per work item. (The
// job engine keeps 2^20: with several jobs in flight a larger pool only mixes
// their scenes, 180 ms against 219 with 2^22 for twelve previews.)
//
// The memory is not the render's alone: a pool above 2^20 slots is halved until
// it fits an eighth of what the device has free (the pool already held counts
// as free) and the caller's budget.
constexpr uint32_t kDefaultSlots = 1u << 24, kSmallPoolSlots = 1u << 20;
constexpr size_t kPoolShare = 8;
inline uint32_t default_slots(uint32_t items, size_t room, size_t budget)
{
    const size_t most = budget ? std::min(room / kPoolShare, budget) : room / kPoolShare;
    uint32_t s = std::max(32u, std::min(kDefaultSlots, items));
    while (s > kSmallPoolSlots && pool_bytes(s) > most)
        s = std::max(kSmallPoolSlots, s / 2);
    return s;
}

// Numbers of slots that vvpt_autotune tries for a render of `items` work items:
// below the default's where it has more, and the default's steps above 2^21 for
// a tuning that starts from a smaller number. As many slots as items or more
// are all the same render.
inline std::vector<uint32_t> autotune_slots(uint32_t items)
{
    std::vector<uint32_t> v{1u << 19, 1u << 20, 3u << 19, 1u << 21, 1u << 22, kDefaultSlots};
    v.erase(std::remove_if(v.begin(), v.end(), [items](uint32_t s) { return s >= items; }), v.end());
    return v;
}

// The memory of one context's renders, kept between them. Other allocations that
// find no room take it back while no render runs (Pools::reclaim).
// Mem: static void *alloc(size_t) (null: no room), void free(void *), size_t
// free_bytes(), int device().
template <class Mem>
class SlotPool {
public:
    // Slots for a render of `items` work items; `wanted` is an explicit number of
    // slots or 0. The pool stays in use until done(). 0: no room (and not in use).
    uint32_t acquire(uint32_t items, uint32_t wanted, size_t budget)
    {
        {
            std::lock_guard<std::mutex> lk(m_mu);
            m_busy = true;
        }
        const uint32_t most = std::max(32u, std::min(wanted ? wanted : kDefaultSlots, items));
        if (m_slots >= most)
            return most;
        // A pool that grows beyond 2^20 slots leaves the old one alone until it
        // is there, and asks nobody else for room.
        if (!wanted && most > kSmallPoolSlots) {
            const uint32_t aim = default_slots(items, Mem::free_bytes() + (m_slots ? pool_bytes(m_slots) : 0), budget);
            for (uint32_t s = aim; s > std::max(m_slots, kSmallPoolSlots); s = std::max(kSmallPoolSlots, s / 2))
                if (void *p = Mem::alloc(pool_bytes(s))) {
                    replace(p, s);
                    return s;
                }
        }
        const uint32_t least = wanted ? most : std::min(most, kSmallPoolSlots);
        if (m_slots >= least)
            return std::min(m_slots, most);
        replace(nullptr, 0);
        void *p = Mem::alloc_or_reclaim(pool_bytes(least));
        if (!p) {
            done();
            return 0;
        }
        replace(p, least);
        return least;
    }
    void done()
    {
        std::lock_guard<std::mutex> lk(m_mu);
        m_busy = false;
    }
    // Frees the memory unless a render uses it; whether there was any. A pool of
    // at most `keep` bytes stays.
    bool give_back(size_t keep = 0)
    {
        std::lock_guard<std::mutex> lk(m_mu);
        if (m_busy || !m_ptr || pool_bytes(m_slots) <= keep)
            return false;
        replace(nullptr, 0);
        return true;
    }
    void *ptr() const { return m_ptr; }
    uint32_t slots() const { return m_slots; } // what the memory holds

    SlotPool() = default;
    SlotPool(const SlotPool &) = delete;
    SlotPool &operator=(const SlotPool &) = delete;
    ~SlotPool() { replace(nullptr, 0); }

private:
    void replace(void *p, uint32_t slots)
    {
        if (m_ptr)
            Mem::free(m_ptr);
        m_ptr = p;
        m_slots = slots;
    }
    std::mutex m_mu; // m_busy; the memory while it is not in use
    bool m_busy = false;
    void *m_ptr = nullptr;
    uint32_t m_slots = 0;
};

// The pools of all contexts of the process.
template <class Mem>
class Pools {
public:
    void add(SlotPool<Mem> *p, int device)
    {
        std::lock_guard<std::mutex> lk(m_mu);
        m_pools.push_back({p, device});
    }
    void remove(SlotPool<Mem> *p)
    {
        std::lock_guard<std::mutex> lk(m_mu);
        m_pools.erase(std::remove_if(m_pools.begin(), m_pools.end(), [p](const Entry &e) { return e.pool == p; }),
                      m_pools.end());
    }
    // Gives back the idle pools of a device; whether that freed anything.
    bool reclaim(int device)
    {
        std::lock_guard<std::mutex> lk(m_mu);
        bool any = false;
        for (const Entry &e : m_pools)
            if (e.device == device)
                any |= e.pool->give_back();
        return any;
    }

private:
    struct Entry {
        SlotPool<Mem> *pool;
        int device;
    };
    std::mutex m_mu;
    std::vector<Entry> m_pools;
};

}  // namespace vvpt
