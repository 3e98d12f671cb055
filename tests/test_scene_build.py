"""Scene creation: meshes packed and instances flattened on the device against
the host's path (bit for bit), runs of faces longer than one core's share,
instances without triangles, and the first bad face of a scene reported."""
import numpy as np
import pytest

from raymond_b200 import api, scenes
from raymond_b200._abi import SceneDesc

pytestmark = pytest.mark.gpu


def _shape(rng, faces, spare_vertices=0):
    v = rng.uniform(-1, 1, (3 * faces + spare_vertices, 3)).astype(np.float32)
    return {"vertices": v, "normals": v.copy(), "texcoords": np.zeros((len(v), 2), np.float32),
            "indices": np.arange(3 * faces, dtype=np.uint32).reshape(-1, 3), "materials": np.zeros(faces, np.uint16)}


def _scene(shapes, entities):
    sc = scenes.cornell(seed=1, envmap_exponent=2)
    vis = sc["entities"][0]["visibility"]
    sc["shapes"] = shapes
    sc["entities"] = [{"shape": s, "matrix": m, "visibility": vis} for s, m in entities]
    return sc


@pytest.mark.parametrize("faces", [1, 2, 65_536, 65_537])
def test_device_and_host_triangles(gpu_ctx, faces):
    rng = np.random.default_rng(faces)
    shapes = [_shape(rng, faces, 3), _shape(rng, 0, 4), _shape(rng, 5)]
    mats = [scenes.translate_scale_rotate_y(rng.uniform(-3, 3, 3), rng.uniform(0.2, 2, 3), a) for a in (0.3, -1.1, 2.0, 0.7)]
    desc = SceneDesc(_scene(shapes, [(1, mats[0]), (0, mats[1]), (1, mats[2]), (2, mats[3]), (0, mats[0]), (1, mats[1])]))
    tris = []
    for builder in ("host", "gpu"):
        sc = api.Scene(api.Context(0, bvh_builder=builder), desc)
        assert sc.info()["triangles"] == 2 * faces + 5
        t = sc.bvh_arrays()[1].view(np.uint32)
        tris.append(t[np.lexsort((t[:, 7], t[:, 3]))])  # by instance and primitive
    assert np.array_equal(*tris)


def test_first_bad_face_is_reported(gpu_ctx):
    rng = np.random.default_rng(1)
    eye = np.eye(4)

    def error(shapes):
        with pytest.raises(api.RmdError) as e:
            api.Scene(gpu_ctx, SceneDesc(_scene(shapes, [(0, eye)])))
        return str(e.value)

    good, index, material = _shape(rng, 70_000), _shape(rng, 70_000), _shape(rng, 9)
    index["indices"][69_999, 1] = 210_000
    material["materials"][3] = 999
    assert "vertex index out of range in shape 1" in error([good, index, material])
    assert "face material out of range in shape 1" in error([good, material, index])
    both = _shape(rng, 70_000)
    both["materials"][66_000] = 999
    both["indices"][66_001, 0] = 210_000
    assert "face material out of range in shape 0" in error([both])
