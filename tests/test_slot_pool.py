"""Sizes of the path-slot pools (csrc/slot_pool.h), compiled for the host."""
import os
import subprocess
import textwrap
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def run_host(tmp_path, body):
    """Output of a program that has slot_pool.h and `body` as its main."""
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                 if p and (Path(p) / "include" / "vector_types.h").exists()), None)
    if not cuda:
        pytest.skip("CUDA headers (vector_types.h) not found")
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text("#include <cstdio>\n#include <vector>\n#include \"slot_pool.h\"\nusing namespace vvpt;\n"
                   + textwrap.dedent(body))
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-I", f"{cuda}/include", "-I", str(ROOT / "include"), "-I",
                    str(ROOT / "vviewer_gb300" / "csrc"), str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()


def test_a_pool_takes_no_more_than_its_paths_members(tmp_path):
    """What the engine's budget and the fixed scratch grant, by the members'
    252 bytes, covers the records of the slots used, and at most one slot in
    64 (or none, of few) is given up."""
    out = run_host(tmp_path, """
        int main()
        {
            std::vector<uint32_t> sizes{32, 33, 63, 64, 65, 1000, 1u << 20, 3u << 19, (1u << 24) - 1, 1u << 24, 1u << 31};
            for (uint32_t s = 32; s < 5000; s++)
                sizes.push_back(s);
            for (uint32_t s : sizes) {
                const uint32_t used = slots_within_members(s);
                const size_t members = 14 * ((16 * (size_t)s + 255) / 256 * 256) + 7 * ((4 * (size_t)s + 255) / 256 * 256);
                if (path_state_bytes(used) > members || used > s || used < s - s / 64 || used < 32)
                    std::printf("%u\\n", s);
            }
            std::printf("%u %u\\n", slots_within_members(1u << 20), slots_within_members(65536));
        }""")
    assert out == [str((1 << 20) * 63 // 64), "64512"], out


FAKE = """
    // A device of 512 MiB to 64 GiB whose allocations are counted.
    struct Mem {
        static size_t total, used;
        static int failed, wide;
        static std::vector<std::pair<char *, size_t>> live;
        static Pools<Mem> pools;
        static void *alloc(size_t n)
        {
            if (used + n > total || (wide && n > (size_t)wide << 20)) {
                failed++;
                return nullptr;
            }
            used += n;
            live.push_back({new char, n});
            return live.back().first;
        }
        static void *alloc_or_reclaim(size_t n)
        {
            void *p = alloc(n);
            return p || !pools.reclaim(0) ? p : alloc(n);
        }
        static void free(void *p)
        {
            for (size_t k = 0; k < live.size(); k++)
                if (live[k].first == p) {
                    used -= live[k].second;
                    delete live[k].first;
                    live.erase(live.begin() + k);
                    return;
                }
            std::printf("free of unknown memory\\n");
        }
        static size_t free_bytes() { return total - used; }
    };
    size_t Mem::total, Mem::used;
    int Mem::failed, Mem::wide; // wide: the largest allocation that succeeds, in MiB (0: any)
    std::vector<std::pair<char *, size_t>> Mem::live;
    Pools<Mem> Mem::pools;
    constexpr size_t GiB = (size_t)1 << 30;
    void device(size_t total, size_t others, int wide = 0)
    {
        Mem::total = total;
        Mem::used = others;
        Mem::failed = 0;
        Mem::wide = wide;
    }
"""


def test_automatic_pool_follows_the_free_memory(tmp_path):
    """At most an eighth of the free memory and the budget above 2^20 slots;
    2^20 slots (or one per work item) whatever is free; never more than the
    work items; an explicit number as it is or not at all."""
    out = run_host(tmp_path, FAKE + """
        uint32_t pool(size_t total, size_t others, uint32_t items, uint32_t wanted = 0, size_t budget = 0)
        {
            device(total, others);
            SlotPool<Mem> p;
            const uint32_t s = p.acquire(items, wanted, budget);
            p.done();
            return s;
        }
        int main()
        {
            const uint32_t many = 50000000;
            std::printf("%u %u %u %u ", pool(280 * GiB, 0, many), pool(64 * GiB, 0, many), pool(64 * GiB, 60 * GiB, many),
                        pool(64 * GiB, 64 * GiB - pool_bytes(1 << 20), many));
            std::printf("%u %u ", pool(64 * GiB, 64 * GiB - pool_bytes(1 << 20) + 1, many), pool(280 * GiB, 0, 3000000));
            std::printf("%u %u %u ", pool(280 * GiB, 0, many, 0, GiB), pool(280 * GiB, 0, many, 0, 1), pool(280 * GiB, 0, 7));
            std::printf("%u %u %u\\n", pool(280 * GiB, 0, many, 1 << 25), pool(8 * GiB, 0, many, 1 << 25),
                        pool(8 * GiB, 0, many, 5000));
        }""")
    # 64 GiB: 5.1 of 8 GiB; 4 GiB free: 0.5 GiB hold 2^20 (0.3 GB) and not 2^21
    assert out == [str(x) for x in (1 << 24, 1 << 24, 1 << 20, 1 << 20, 0, 3000000, 1 << 21, 1 << 20, 32, 1 << 25, 0,
                                    5000)]


def test_pool_is_kept_given_back_and_never_lost_to_a_larger_one(tmp_path):
    out = run_host(tmp_path, FAKE + """
        int main()
        {
            const uint32_t many = 50000000;
            // growth that fails keeps the pool that is there, and is not tried
            // again and again down to nothing
            device(280 * GiB, 0, 400); // no allocation above 400 MiB succeeds
            {
                SlotPool<Mem> p;
                const uint32_t a = p.acquire(many, 0, 0);
                p.done();
                const void *at = p.ptr();
                const uint32_t b = p.acquire(many, 0, 0);
                p.done();
                std::printf("%u %u %d ", a, b, (int)(p.ptr() == at));
            }
            // in use: not given back; idle: given back to another allocation, and
            // made again by the next render
            device(64 * GiB, 0);
            SlotPool<Mem> p, q;
            Mem::pools.add(&p, 0);
            Mem::pools.add(&q, 1);
            const uint32_t a = p.acquire(many, 0, 0);
            const bool busy = Mem::pools.reclaim(0);
            p.done();
            q.acquire(1000, 0, 0);
            q.done();
            void *other = Mem::alloc_or_reclaim(60 * GiB); // needs p's 4.7 GiB
            std::printf("%u %d %d %u %u ", a, (int)busy, (int)(other != nullptr), p.slots(), q.slots());
            const uint32_t small = p.acquire(many, 0, 0); // an eighth of 4 GiB is free
            p.done();
            Mem::free(other);
            const uint32_t large = p.acquire(many, 0, 0);
            p.done();
            std::printf("%u %u ", small, large);
            // a smaller explicit number: above it the memory goes back
            const bool kept = !p.give_back(pool_bytes(1 << 24)), freed = p.give_back(pool_bytes(1 << 20));
            std::printf("%d %d %u ", (int)kept, (int)freed, p.acquire(many, 1 << 20, 0));
            p.done();
            // a smaller render in a larger pool uses its own items
            std::printf("%u %zu\\n", p.acquire(77, 0, 0), Mem::live.size());
            p.done();
            Mem::pools.remove(&p);
            std::printf("%d\\n", (int)Mem::pools.reclaim(0));
        }""")
    assert out == [str(x) for x in (1 << 20, 1 << 20, 1, 1 << 24, 0, 1, 0, 1000, 1 << 20, 1 << 24, 1, 1, 1 << 20, 77, 2,
                                    0)]


def test_blocks_per_sm_reach_every_kernel(tmp_path):
    """A caller's blocks_per_sm is every kernel's grid, up to one thread per
    slot; the default keeps to the blocks that run at once."""
    out = run_host(tmp_path, """
        int main()
        {
            for (int automatic = 0; automatic < 2; automatic++)
                for (int per_sm : {2, 8}) {
                    const LaunchShape s{152 * 6, 256, 152, 1u << 24, automatic != 0}, few{152 * 6, 128, 152, 1000,
                                                                                                  automatic != 0};
                    std::printf("%d %d\\n", launch_blocks(s, s.grid, per_sm, 256), launch_blocks(few, few.grid, per_sm, 128));
                }
        }""")
    assert out == ["912", "8", "912", "8", "304", "8", "912", "8"]


def test_autotuner_tries_slots_up_to_the_default(tmp_path):
    out = run_host(tmp_path, """
        int main()
        {
            for (uint32_t items : {1u, 1u << 19, (1u << 20) + 1, 33000000u}) {
                for (uint32_t s : autotune_slots(items))
                    std::printf("%u,", s);
                std::printf("end\\n");
            }
        }""")
    small = f"{1 << 19},{1 << 20},"
    assert out == ["end", "end", small + "end", small + f"{3 << 19},{1 << 21},{1 << 22},{1 << 24},end"]
