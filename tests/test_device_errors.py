"""A device error ends a render within a few iterations (host side, the device's part played by the test)."""
import numpy as np
import pytest

from host_runtime import ERRORS, PATHS_DONE, fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc

W, H, SPP, POOL = 64, 48, 64, 64  # 3,072 pools of paths


def _render(fake, call, see_counters, also=lambda *call: 0):
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    ctx = api.Context(0)
    if call == "batch":
        b = api.Batch(ctx, [desc], [{"scene": 0, "width": W, "height": H}], pool_size=POOL, graph=False)
        run = lambda: b.render(spp=SPP, max_depth=4, first_sample=0)
    elif call == "noalloc":
        scene, film = api.Scene(ctx, desc), np.zeros((H, W, 4), np.float32)
        run = lambda: api.render_noalloc(scene, desc.scene["camera"], W, H, film.ctypes.data, spp=SPP, first_sample=0,
                                         max_depth=4, pool_size=POOL)
    else:
        r = api.Renderer(api.Scene(ctx, desc), W, H, pool_size=POOL)
        if call == "guided":
            r.set_guide(sampling=True, training=False)
        run = lambda: r.render(spp=SPP, max_depth=4, first_sample=0)
    iterations = [0]

    def see(name, ptr, size, stream):
        if name == "launch:rmd_shade":
            iterations[0] += 1
        elif fake.is_counters(name, size):
            fake.counter(ptr, ERRORS, 32).value = 0  # the kernel that clears them does nothing here
            see_counters(ptr, iterations[0])
        return also(name, ptr, size, stream)

    with fake.on(see):
        run()
    return iterations[0]


@pytest.mark.parametrize("call", ["render", "guided", "noalloc", "batch"])
def test_errors_are_seen_early(fake, call):
    seen = []

    def error(ptr, iterations):
        seen.append(iterations)
        fake.counter(ptr, ERRORS, 32).value = 2

    with pytest.raises(fake.api.RmdError, match="error flags"):
        _render(fake, call, error)
    assert seen[0] <= 16 and seen[-1] <= 32


@pytest.mark.parametrize("call", ["render", "noalloc", "batch"])
@pytest.mark.parametrize("ends", [3074, 3081, 4000])
def test_the_end_is_seen_soon(fake, call, ends):
    """A render ends within six iterations of its last path (the counters of iteration i are read after i + 2)."""
    def play(ptr, iterations):
        fake.counter(ptr, PATHS_DONE).value = W * H * SPP if iterations >= ends else 0

    assert ends <= _render(fake, call, play) <= ends + 6


@pytest.mark.parametrize("call", ["render", "guided", "noalloc", "batch"])
def test_a_failed_launch_is_reported_once(fake, call):
    """The error of a launch that fails is its call's; the next calls succeed."""
    launches = 0

    def see(name, ptr, size, stream):
        nonlocal launches
        if name.startswith("launch:"):
            launches += 1
            return 98 if launches == 6 else 0  # cudaErrorInvalidDeviceFunction

    with pytest.raises(fake.api.RmdError, match="CUDA error 98"):
        _render(fake, call, lambda ptr, iterations: None, also=see)
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    fake.api.Scene(fake.api.Context(0), desc).close()


@pytest.mark.parametrize("call", ["render", "guided", "trained", "noalloc", "batch", "graph"])
def test_a_failed_call_leaves_no_work_behind(fake, call):
    """When a launch fails, what was enqueued before has ended on return: the objects may go at once."""
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    ctx = api.Context(0)
    if call in ("batch", "graph"):
        x = api.Batch(ctx, [desc], [{"scene": 0, "width": W, "height": H}], pool_size=POOL, graph=call == "graph")
    else:
        scene, film = api.Scene(ctx, desc), np.zeros((H, W, 4), np.float32)
        x = api.Renderer(scene, W, H, pool_size=POOL)
        if call in ("guided", "trained"):
            x.set_guide(sampling=call == "guided", training=call == "trained")
    streams, launches = set(), 0

    def see(name, ptr, size, stream):
        nonlocal launches
        if stream:
            streams.add(stream)
        if name.startswith("launch:") or name == "cudaGraphLaunch":
            launches += 1
            if launches == (2 if call == "graph" else 12):
                return 98  # cudaErrorInvalidDeviceFunction

    with fake.on(see), pytest.raises(api.RmdError, match="CUDA error 98"):
        if call == "noalloc":
            api.render_noalloc(scene, desc.scene["camera"], W, H, film.ctypes.data, spp=SPP, first_sample=0, max_depth=4)
        else:
            x.render(spp=SPP, max_depth=4, first_sample=0)
    assert streams and [fake.lib.fake_pending(s) for s in streams] == [0] * len(streams)
    x.close()
