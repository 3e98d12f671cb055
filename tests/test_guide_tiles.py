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


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 127, 128, 129, 4099, 64 * 128 + 77])
def test_gradient_sizes_match_oracle(gpu_ctx, n):
    """The training kernel's gradient at tile edges (128 records per CTA; the
    padding rows of a last tile) and with several tiles per CTA, per layer:
    cosine above 0.998 and norm within 3 % of the float64 oracle's."""
    rng = np.random.default_rng(n)
    params = G.init_params(2)
    params[-G.OUTPUTS:] += rng.normal(0, 0.5, G.OUTPUTS).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    rec = np.concatenate([rng.uniform(0, 1, (n, 7)), d, rng.uniform(0.05, 0.6, (n, 1)), rng.gamma(0.5, 1.0, (n, 1))],
                         axis=1).astype(np.float32)
    grad, loss = api.guide_gradient(params, rec)
    want_loss, want = G.loss_and_grad(params, rec)
    assert abs(loss - want_loss) <= 1e-3 * abs(want_loss) + 1e-4
    off = 0
    for i, o in G.LAYERS:
        for k in (i * o, o):
            g, c = grad[off:off + k], want[off:off + k]
            assert g @ c > 0.998 * np.linalg.norm(g) * np.linalg.norm(c)
            assert abs(np.linalg.norm(g) / np.linalg.norm(c) - 1) <= 0.03
            off += k
