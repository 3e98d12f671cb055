"""The device builder's clustering at its edges: cluster counts around a
block's threads, around the count from which one block goes on alone, and
beyond one run of clusters per block, with triangles that all cost the same
among them (merged pairwise)."""
import numpy as np
import pytest

from test_bvh_gpu import both, check_tree, random_rays, same_hits, soup_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 511, 512, 513, 1025, 4097, 160_001])
@pytest.mark.parametrize("kind", ["random", "identical"])
def test_cluster_counts(gpu_ctx, n, kind):
    rng = np.random.default_rng(n)
    v = rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))
    if kind == "identical":
        v[:] = v[0]
    host, gpu = both(soup_scene(v))
    raw, tris = gpu.bvh_arrays()
    assert len(tris) == n and gpu.bvh_stats()["levels"] <= 32
    if n < 10_000:
        check_tree(raw, tris)
    key = lambda t: np.lexsort((t[:, 7].view(np.uint32), t[:, 3].view(np.uint32)))
    htris = host.bvh_arrays()[1]
    assert np.array_equal(tris[key(tris)], htris[key(htris)])
    rays = random_rays(np.random.default_rng(5), v.min() - 0.5, v.max() + 0.5, 2000 if kind == "identical" else 20000)
    same_hits(host, gpu, rays)
