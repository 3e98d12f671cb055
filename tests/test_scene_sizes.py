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
