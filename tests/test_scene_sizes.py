"""Scene creation at the ends of its counters (host side)."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from host_runtime import ROOT, fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc


@pytest.mark.parametrize("entities", [17, 4097])
def test_more_triangles_than_the_device_builder_takes(fake, entities):
    """Refused for their number, before anything is allocated for them."""
    api = fake.api
    faces = 1 << 20
    sc = scenes.cornell(seed=1, envmap_exponent=2)
    vis = sc["entities"][0]["visibility"]
    sc["shapes"] = [{"vertices": np.zeros((3, 3), np.float32), "normals": np.zeros((3, 3), np.float32),
                     "texcoords": np.zeros((3, 2), np.float32), "indices": np.zeros((faces, 3), np.uint32),
                     "materials": np.zeros(faces, np.uint16)}]
    sc["entities"] = [{"shape": 0, "matrix": np.eye(4), "visibility": vis}] * entities
    asked = []

    def see(name, ptr, size, stream):
        if name == "cudaMalloc":
            asked.append(size)

    with fake.on(see), pytest.raises(api.RmdError, match="INVALID_ARGUMENT.*takes at most 2\\^24 triangles"):
        api.Scene(api.Context(0, bvh_builder="gpu"), SceneDesc(sc))
    assert max(asked) < 64 << 20  # the mesh's own arrays


COUNTS = [0, 1, 65_535, 65_536, 65_537, 3 * 65_536, 0xFFFF_0000, 0xFFFF_0001, 0xFFFF_FFFF]


def test_runs_of_faces_end(tmp_path):
    """The runs that the cores check cover a shape's faces once, to the largest 32-bit count."""
    src = tmp_path / "runs.cpp"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include "face_runs.h"\n'
                   "int main(int argc, char **argv) {\n"
                   "    for (int k = 1; k < argc; k++) {\n"
                   "        std::vector<rmdhost::FaceRun> runs;\n"
                   "        rmdhost::appendFaceRuns(runs, k, (uint32_t)std::strtoul(argv[k], nullptr, 10));\n"
                   "        unsigned long long at = 0;\n"
                   "        for (const auto &r : runs) {\n"
                   "            if (r.shape != k || r.begin != at || r.end < r.begin || r.end - r.begin > 65536) return 1;\n"
                   "            at = r.end;\n"
                   "        }\n"
                   '        std::printf("%llu %zu\\n", at, runs.size());\n'
                   "    }\n}\n")
    exe = tmp_path / "runs"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(ROOT / "raymond_b200" / "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), *map(str, COUNTS)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert [tuple(map(int, line.split())) for line in out.splitlines()] == [(n, max(1, -(-n // 65_536))) for n in COUNTS]


@pytest.mark.parametrize("vertices,faces", [(3, 1), (0, 0xFFFF_FFFF), (0xFFFF_FFFF, 3)])
def test_meshes_are_packed_by_a_grid(fake, vertices, faces):
    """The packing kernel's grid at the largest 32-bit counts (no kernel runs here)."""
    names = subprocess.run(["nm", "-D", "--defined-only", str(fake.path)], check=True, capture_output=True, text=True).stdout
    pack = fake.lib[next(n for n in names.split() if "rmdLaunchPackMesh" in n)]
    p, grids = C.c_void_p(0), []
    pack.argtypes = [C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.c_void_p, C.c_uint64] + [C.c_void_p] * 4

    def see(name, ptr, size, stream):
        if "k_pack_mesh" in name:
            grids.append(size)

    with fake.on(see):
        assert pack(p, p, vertices, p, p, faces, p, p, p, p) == 0
    assert len(grids) == 1 and 1 <= grids[0] <= 148 * 16
