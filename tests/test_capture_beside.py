"""Objects that go while another thread captures a graph (a batch does when it
first renders with new settings; a host program may at any time): a wait for the
whole device is refused then and spoils the capture."""
import threading
import time

import numpy as np
import pytest

from host_runtime import fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc

VIEWS = [{"scene": 0, "width": 24, "height": 16}]


def test_destruction_waits_for_no_device(fake):
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    ctx = api.Context(0)
    streams, calls = [], []

    def see(name, ptr, size, stream):
        calls.append(name)
        if name == "cudaMemsetAsync":
            streams.append(stream)

    scene = api.Scene(ctx, desc)
    r = api.Renderer(scene, 24, 16, pool_size=2048)
    r.set_guide(sampling=True, training=True, replay_records=1 << 12)
    b = api.Batch(ctx, [desc], VIEWS, pool_size=2048)
    with fake.on(see):
        other = api.Renderer(api.Scene(api.Context(0), desc), 24, 16, pool_size=2048)  # whose stream is captured
    fake.lib.fake_set_capturing(streams[-1], 1)
    calls.clear()
    with fake.on(see):
        r.close(), b.close(), scene.close()
    fake.lib.fake_set_capturing(streams[-1], 0)
    other.close()
    assert "cudaDeviceSynchronize" not in calls and "cudaStreamSynchronize" not in calls


@pytest.mark.gpu
def test_batches_beside_renderers_that_go(gpu_ctx):
    """Batches captured anew on every render while another thread makes and drops scenes and renderers."""
    from raymond_b200 import api

    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=4))
    batch = api.Batch(gpu_ctx, [desc], VIEWS, pool_size=1 << 12)

    def render(depth):
        batch.reset()
        batch.render(spp=1, max_depth=depth, first_sample=0)
        return batch.film(0)

    alone = {d: render(d) for d in (2, 3, 4, 5)}
    stop, failed, made = threading.Event(), [], [0]

    def objects():
        try:
            ctx = api.Context(0)
            while not stop.is_set():
                scene = api.Scene(ctx, desc)
                r = api.Renderer(scene, 16, 16, pool_size=1 << 10)
                r.render(spp=1, max_depth=2)
                r.close(), scene.close()
                made[0] += 1
        except Exception as e:  # reported by the main thread
            failed.append(e)

    t = threading.Thread(target=objects)
    t.start()
    try:
        films, until = [], time.monotonic() + 120  # the other thread may have to compile its module first
        while (len(films) < 240 or made[0] < 4) and not failed and time.monotonic() < until:
            films += [(d, render(d)) for d in (2, 3, 4, 5)]
    finally:
        stop.set()
        t.join()
    assert not failed and made[0] > 3
    for d, f in films:
        np.testing.assert_array_equal(f, alone[d])


def test_a_batch_captures_on_a_stream_of_its_own(fake):
    """What other threads enqueue on the context's stream meanwhile is not captured with it."""
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    ctx = api.Context(0)
    b = api.Batch(ctx, [desc], VIEWS, pool_size=2048)
    r = api.Renderer(api.Scene(ctx, desc), 24, 16, pool_size=2048)
    captured, launched, during = [], [], []

    def see(name, ptr, size, stream):
        if name == "cudaStreamBeginCaptureToGraph":
            captured.append(stream)
        elif name == "cudaGraphLaunch":
            launched.append(stream)
        elif name == "launch:rmd_shade" and captured and not launched:
            during.append(stream)
            r.reset()  # clears its film on the context's stream and waits for it

    with fake.on(see):
        b.render(spp=1, max_depth=2, first_sample=0)
        b.render(spp=1, max_depth=3, first_sample=0)
    assert len(captured) == len(launched) == 2 and during and set(during) <= set(captured)
    assert not set(captured) & set(launched)
    r.close(), b.close()
