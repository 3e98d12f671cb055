"""Counters and films are cleared in the order of the context's stream: new
buffers may be kept blocks that hold an earlier object's contents, and the
legacy stream is not ordered with the context's."""
import numpy as np
import pytest

from host_runtime import fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc

VIEWS = [{"scene": 0, "width": 24, "height": 16}, {"scene": 0, "width": 9, "height": 31}]


def test_no_clear_on_the_legacy_stream(fake):
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    clears = []

    def see(name, ptr, size, stream):
        if name == "cudaMemset" or (name == "cudaMemsetAsync" and not stream):
            clears.append((name, size))

    with fake.on(see):
        ctx = api.Context(0)
        scene = api.Scene(ctx, desc)
        r = api.Renderer(scene, 24, 16, pool_size=2048)
        r.set_tuning({"shade_min_blocks": 5, "trace_blocks_per_sm": 8, "pool_size": 4096})
        r.set_guide(sampling=True, training=True, batch_size=1 << 12, replay_records=1 << 12)
        r.set_guide(sampling=True, training=True, reset=True, replay_records=1 << 13)
        scene.trace(np.zeros((3, 8), np.float32))
        b = api.Batch(ctx, [desc], VIEWS, pool_size=2048)
        b.set_guide(sampling=True, training=True, replay_records=1 << 12)
    assert clears == []
    assert fake.lib.fake_pending(None) == 0


@pytest.mark.gpu
def test_clears_beside_a_busy_default_stream(gpu_ctx):
    """With milliseconds of work queued on the default stream, a new pool or batch renders what it renders otherwise."""
    import torch

    from raymond_b200 import api

    desc = SceneDesc(scenes.cornell(seed=2, envmap_exponent=4))
    scene = api.Scene(gpu_ctx, desc)
    a = torch.randn(4096, 4096, device="cuda")

    def busy():
        x = a
        for _ in range(20):
            x = a @ x * 1e-2

    def pool(size, load):
        r = api.Renderer(scene, 48, 40)
        r.render(spp=1, max_depth=6, first_sample=0)
        r.reset()
        if load:
            busy()
        r.set_tuning({"shade_min_blocks": 5, "trace_blocks_per_sm": 12, "pool_size": size})
        r.render(spp=1, max_depth=6, first_sample=0)
        return r.film()

    def batch(load):
        b = api.Batch(gpu_ctx, [desc], VIEWS, pool_size=1 << 12)
        b.render(spp=1, max_depth=6, first_sample=0)  # leaves its film and counters among the kept blocks
        del b
        if load:
            busy()
        b = api.Batch(gpu_ctx, [desc], VIEWS, pool_size=1 << 12)
        b.render(spp=1, max_depth=6, first_sample=0)
        return [b.film(v) for v in range(len(VIEWS))]

    want = pool(1 << 14, False), batch(False)
    for _ in range(5):
        np.testing.assert_array_equal(pool(1 << 14, True), want[0])
        for x, y in zip(batch(True), want[1]):
            np.testing.assert_array_equal(x, y)
        torch.cuda.synchronize()
