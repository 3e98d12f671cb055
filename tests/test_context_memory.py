"""A context hands the blocks of objects that went to the next ones."""
import numpy as np
import pytest

from raymond_b200 import api, scenes
from raymond_b200._abi import SceneDesc


@pytest.mark.gpu
@pytest.mark.parametrize("builder", ["host", "gpu"])
def test_kept_blocks_leave_images_as_they_are(builder):
    """Scenes and renderers of alternating sizes, created and dropped in one
    context, render what a context of their own renders, bit for bit."""
    cases = [(scenes.spheres_terrain(seed=k, num_spheres=4 + k, subdivisions=1 + k % 2, terrain_cells=8 + 3 * k), 40 + 8 * k)
             for k in range(4)]

    def render(ctx, desc, width):
        r = api.Renderer(api.Scene(ctx, SceneDesc(desc)), width, 32, pool_size=1 << (10 + width % 3))
        r.render(spp=2, max_depth=4, film_fp64=True)
        return r.film64()

    shared = api.Context(0, bvh_builder=builder)
    for k in (0, 3, 1, 2, 0, 2, 3):
        np.testing.assert_array_equal(render(shared, *cases[k]), render(api.Context(0, bvh_builder=builder), *cases[k]))
