"""Rays traced by groups of 8 lanes (few rays in flight) against rays traced by
whole warps, and small pools against large ones: each path's arithmetic is the
same, so at one sample per pixel (one addition per pixel) the films of a pool
of a few paths, whose rays are all traced by groups, and of the default pool
are equal bit for bit, and so are the ray counts."""
import numpy as np
import pytest

from raymond_b200 import api, scenes
from raymond_b200._abi import RNG_TEA, SAMPLING_BSDF, SAMPLING_MIS, SAMPLING_NEE, SceneDesc

pytestmark = pytest.mark.gpu


def _scene(name):
    if name == "lights":
        return scenes.cornell_all_lights(seed=5)
    if name == "terrain":
        return scenes.spheres_terrain(seed=2, num_spheres=16, subdivisions=3, terrain_cells=48, envmap_exponent=5)
    sc = scenes.cornell(seed=3, envmap_exponent=4)
    if name == "empty":  # no triangle: every ray misses
        sc["entities"] = []
    return sc


# one path, around a group's warp and block, more paths than are traced by groups (28 k rays)
SIZES = [(1, 1), (3, 1), (5, 1), (17, 1), (13, 5), (257, 1), (301, 126), (401, 233)]


@pytest.mark.parametrize("name", ["cornell", "lights", "terrain", "empty"])
def test_groups_equal_warps(gpu_ctx, name):
    scene = api.Scene(gpu_ctx, SceneDesc(_scene(name)))
    for (w, h), mode, kw in zip(SIZES, [SAMPLING_MIS, SAMPLING_NEE, SAMPLING_BSDF, SAMPLING_MIS] * 2,
                                [{}, {"rng": RNG_TEA}, {"film_fp64": True}, {}] * 2):
        got = []
        for pool in (max(1, min(4096, w * h // 8)), 0):
            r = api.Renderer(scene, w, h, pool_size=pool)
            r.render(spp=1, max_depth=9, sampling_mode=mode, first_sample=2, **kw)
            st = r.stats()
            assert st["paths"] == w * h and st["rays"] >= w * h and st["errors"] == 0
            got.append((r.film64() if kw.get("film_fp64") else r.film(),
                        [st[k] for k in ("segments", "rays", "shadow_rays")]))
        assert np.array_equal(got[0][0], got[1][0]), (name, w, h)
        assert got[0][1] == got[1][1], (name, w, h)


@pytest.mark.parametrize("graph", [True, False])
def test_groups_in_batches(gpu_ctx, graph):
    """Views of different scenes, each ray with its view's tree."""
    descs = [SceneDesc(_scene("cornell")), SceneDesc(_scene("terrain"))]
    views = [{"scene": 0, "width": 61, "height": 47}, {"scene": 1, "width": 330, "height": 170},
             {"scene": 0, "width": 1, "height": 3}]
    small = api.Batch(gpu_ctx, descs, views, pool_size=1500, graph=graph)
    whole = api.Batch(gpu_ctx, descs, views, graph=graph)
    for b in (small, whole):
        b.render(spp=1, max_depth=8, first_sample=1)
        assert b.stats()["paths"] == 61 * 47 + 330 * 170 + 3
    for v in range(len(views)):
        assert np.array_equal(small.film(v), whole.film(v)), v
