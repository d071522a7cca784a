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
