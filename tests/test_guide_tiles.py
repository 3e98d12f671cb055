"""Sizes at which the guide's inference tiles (128 samples, four pipelines per
CTA) and the interleaved mixtures (32 hits) can go wrong."""
import numpy as np
import pytest

from oracle import guide_mlp as G
from raymond_b200 import api, scenes
from raymond_b200._abi import SceneDesc


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 513, 1025, 148 * 512 + 128 * 5 + 3])
def test_forward_sizes_match_oracle(gpu_ctx, n):
    """Raw outputs against the BF16-emulating oracle, within 2e-3 + 1e-2 |x|
    (hidden activations can round to the next BF16 value); features on bin
    edges, at the ends of [0, 1] and outside it among them."""
    rng = np.random.default_rng(n)
    params = G.init_params(5)
    params[-G.OUTPUTS:] += rng.normal(0, 0.5, G.OUTPUTS).astype(np.float32)
    feats = rng.uniform(0, 1, (n, 7)).astype(np.float32)
    edges = np.array([[0] * 7, [1] * 7, [0.5 / 32] * 7, [0.5 / 16] * 7, [31.5 / 32] * 7, [15.5 / 16] * 7,
                      [-0.01] * 7, [1.01] * 7, [3.0] * 7, [0.25] * 7], np.float32)
    feats[:min(n, 10)] = edges[:min(n, 10)]
    gpu = api.guide_forward(params, feats)
    sel = np.unique(np.r_[np.arange(min(n, 600)), np.arange(max(0, n - 600), n)])
    cpu, _ = G.forward(params, feats[sel])
    err = np.abs(gpu[sel] - cpu)
    assert np.all(err <= 2e-3 + 1e-2 * np.abs(cpu)), float(err.max())


@pytest.mark.gpu
@pytest.mark.parametrize("pool", [33, 1000, 1 << 14])
def test_guided_render_at_pool_sizes(gpu_ctx, pool):
    """Guided renders over pools that are no multiple of 32 or of a tile: the
    mean radiance over 8 seeds is the plain tracer's within 5 standard errors."""
    scene = api.Scene(gpu_ctx, SceneDesc(scenes.cornell(seed=1, envmap_exponent=6)))

    def means(guided):
        out = []
        for seed in range(8):
            r = api.Renderer(scene, 24, 16, pool_size=pool)
            if guided:
                r.set_guide(sampling=True, training=True, batch_size=1 << 12, steps_per_batch=2, seed=3)
            r.render(spp=64, max_depth=6, film_fp64=True, seed=100 + seed)
            out.append(r.film64().mean() / 64)
            assert r.stats()["errors"] == 0
        return np.array(out)
    a, b = means(False), means(True)
    err = np.sqrt((a.var(ddof=1) + b.var(ddof=1)) / 8)
    assert abs(a.mean() - b.mean()) <= 5 * err, (a.mean(), b.mean(), err)
