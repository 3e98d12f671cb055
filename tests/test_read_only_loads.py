"""Loads through the read-only path (__ldg, ld.global.nc) are for data that no
running kernel writes.  Kernels of a render overlap: one is resident before the
kernel ahead has written what it reads, so path state, queues, records and the
guide's network are read by coherent loads; the scene's trees and triangles,
written before any render, may be read either way."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "raymond_b200" / "csrc"
# nodes and triangles (device/traverse.cuh); the read-only arrays of a scene's set-up kernels
TREE = re.compile(r"^(&np->\w+|reinterpret_cast<const uint2 \*>\(&np->bases\)|nb \+ .*|&nodes\[0\]\.\w+|&tv\[[012]\]|"
                  r"&tris\[TRI_FLOAT4 \* \(size_t\)s\.hitTri \+ [67]\])$")


def _arguments(text, call):
    for m in re.finditer(re.escape(call) + r"\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def _code(path):
    text = path.read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def test_only_trees_are_read_through_the_read_only_path():
    files = sorted(CSRC.glob("*.cu")) + sorted((CSRC / "device").glob("*.cuh"))
    found = [(f.name, a) for f in files for a in _arguments(_code(f), "__ldg")]
    assert len(found) > 20
    assert [x for x in found if not TREE.match(x[1])] == []
    assert not any("ld.global.nc" in _code(f) for f in files)


def test_no_restrict_pointer_to_what_a_render_writes():
    """A const __restrict__ parameter lets the compiler take the read-only path by itself."""
    for f in [CSRC / "kernels.cu", CSRC / "guide.cu", *sorted((CSRC / "device").glob("*.cuh"))]:
        for t in re.findall(r"const\s+(\w+)\s*\*\s*__restrict__\s*(\w+)", _code(f)):
            assert t[0] in ("WideNode", "float4", "float", "uint32_t", "uint16_t", "uint4", "PerInstanceData"), (f.name, t)
            assert t[1] in ("nodes", "tris", "sceneNodes", "sceneTris", "in", "pos", "nrm", "idx", "mat", "vertices", "faces",
                            "instances"), (f.name, t)
