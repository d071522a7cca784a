"""Scene packing where the builder outside (the GPU) leaves its meshes to the
host, as it does without room for them: the scene is the host's own. A
failure is still an error."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

from raygen import HIT_SCENES
from vviewer_gb300 import _native as N

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "vviewer_gb300" / "csrc"
HARNESS = Path(__file__).resolve().parent / "host_pack" / "host_pack.cpp"
OUT = Path(__file__).resolve().parent / "_build" / "libhost_pack.so"


@pytest.fixture(scope="module")
def host_lib():
    cuda = next((p for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                 if p and (Path(p) / "include" / "vector_types.h").exists()), None)
    if not cuda:
        pytest.skip("CUDA headers (vector_types.h) not found")
    srcs = [HARNESS, CSRC / "scene_pack.cpp", CSRC / "bvh_build.cpp", CSRC / "bvh_wide.cpp"]
    OUT.parent.mkdir(exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-I",
                    f"{cuda}/include", "-I", str(ROOT / "include"), "-I", str(CSRC), *map(str, srcs), "-o", str(OUT)],
                   check=True, capture_output=True)
    lib = C.CDLL(str(OUT))
    lib.host_pack_status.argtypes = [C.c_void_p, C.c_char_p, C.c_int]
    lib.host_pack_outside.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_int), C.c_char_p, C.c_int]
    return lib


def pack(lib, flat, failure):
    desc, asked, msg = flat.desc(), C.c_int(0), C.create_string_buffer(256)
    return lib.host_pack_outside(C.addressof(desc), failure, C.byref(asked), msg, 256), asked.value, msg.value


@pytest.mark.parametrize("name", ["displaced_spheres", "volume_cube"])
def test_declined_meshes_are_built_on_the_host(host_lib, name):
    flat = HIT_SCENES[name][0]().scene.build()
    large = sum(m.num_triangles >= 100 for m in flat.desc().meshes[:flat.desc().num_meshes])
    assert pack(host_lib, flat, b"") == (0, large, b"")
    if large:
        assert pack(host_lib, flat, b"broken") == (5, large, b"broken")  # VVPT_ERR_DEVICE
    assert name != "displaced_spheres" or large > 0


def test_scenes_beyond_the_reference_bits_are_refused(host_lib):
    """Counts that an index of 30 bits (or 32-bit offsets) cannot name: refused
    before anything is read (the arrays here hold one element)."""
    for meshes, tris, verts in ((1, 1 << 30, 3), (2, (1 << 30) - 1, 3), (3, 1, 1 << 31)):
        vertex, corner = N.Vertex(), (C.c_uint32 * 3)()
        md = (N.MeshDesc * meshes)()
        for m in md:
            m.vertices, m.num_vertices = C.addressof(vertex), verts
            m.indices, m.num_triangles = C.addressof(corner), tris
        desc = N.SceneDesc()
        desc.meshes, desc.num_meshes = md, meshes
        msg = C.create_string_buffer(256)
        assert host_lib.host_pack_status(C.addressof(desc), msg, 256) == 8, msg.value  # VVPT_ERR_UNSUPPORTED
