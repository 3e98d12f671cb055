"""A context's kept blocks and the allocations that find the device full (host
side, on a device whose size the test sets)."""
import subprocess
import sys
from pathlib import Path

import pytest

from host_runtime import OUT_OF_MEMORY, PATHS_DONE, fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc

W, H = 512, 512
DESC = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))


def _full_device(fake, ctx, blocks=3):
    """Blocks of ~0.5 GB kept by `ctx`, and nothing else free on the device."""
    api = fake.api
    scene = api.Scene(ctx, DESC)
    renderers = [api.Renderer(scene, 16, 16, pool_size=1 << 21) for _ in range(blocks)]
    for r in renderers:
        r.close()
    assert fake.lib.fake_allocated() > blocks * (500 << 20)
    fake.lib.fake_set_capacity(fake.lib.fake_allocated() + (1 << 20))
    return scene


def test_film_takes_what_the_context_keeps(fake):
    scene = _full_device(fake, fake.api.Context(0))
    r = fake.api.Renderer(scene, W, H, pool_size=1 << 12)  # 4 MB of film, outside the pool
    r.set_size(2 * W, 2 * H)
    r.close()


def test_network_takes_what_the_context_keeps(fake):
    api = fake.api
    ctx = api.Context(0)
    r = api.Renderer(api.Scene(ctx, DESC), 16, 16, pool_size=1 << 12)
    _full_device(fake, ctx)
    r.set_guide(sampling=True, training=True)  # the gradient slots of the network: 27 MB
    assert len(r.guide_params()) == api.guide_param_count()
    r.close()


def test_another_context_takes_what_a_context_keeps(fake):
    api = fake.api
    scene = _full_device(fake, api.Context(0))
    r = api.Renderer(api.Scene(api.Context(0), DESC), W, H, pool_size=1 << 20)
    r.close(), scene.close()


@pytest.mark.parametrize("call", ["cudaLibraryLoadData", "cudaGraphInstantiate"])
def test_modules_and_graphs_take_what_a_context_keeps(fake, call):
    api = fake.api
    ctx = api.Context(0)
    scene = _full_device(fake, ctx)
    kept = fake.lib.fake_allocated()
    failed = []

    def see(name, ptr, size, stream):
        if name == call and not failed:
            failed.append(fake.lib.fake_allocated())
            return OUT_OF_MEMORY

    with fake.on(see):
        b = api.Batch(ctx, [DESC], [{"scene": 0, "width": 8, "height": 8}], pool_size=1 << 10)
        if call == "cudaGraphInstantiate":
            b.render(spp=1, max_depth=2, first_sample=0)
    assert failed and fake.lib.fake_allocated() < kept - (1 << 30)
    b.close(), scene.close()


def test_out_of_memory_is_reported_when_nothing_is_kept(fake):
    api = fake.api
    scene = api.Scene(api.Context(0), DESC)
    fake.lib.fake_set_capacity(fake.lib.fake_allocated() + (1 << 20))
    with pytest.raises(api.RmdError, match="OUT_OF_MEMORY"):
        api.Renderer(scene, W, H, pool_size=1 << 20)
    fake.lib.fake_set_capacity(180 << 30)
    api.Renderer(scene, W, H, pool_size=1 << 20).close()  # and the failure is forgotten
    scene.close()


def test_the_bound_holds_and_all_goes_with_the_context(fake):
    api = fake.api
    before = fake.lib.fake_allocated()
    ctx = api.Context(0)
    scene = api.Scene(ctx, DESC)
    base = fake.lib.fake_allocated()
    renderers = [api.Renderer(scene, 16, 16, pool_size=1 << 21) for _ in range(6)]
    for r in renderers:
        r.close()
    assert base < fake.lib.fake_allocated() <= base + (2 << 30)
    scene.close()
    ctx.close()
    del scene
    assert fake.lib.fake_allocated() == before


def test_autotune_counts_kept_memory_as_free(fake):
    """Pools are tried if they fit into half of the free memory; blocks that contexts keep are free."""
    api = fake.api
    ctx = api.Context(0)
    scene = api.Scene(ctx, DESC)
    r = api.Renderer(scene, 16, 16, pool_size=1 << 16)
    _full_device(fake, ctx).close()
    tried = []

    def see(name, ptr, size, stream):
        if name == "cudaMalloc" and size > 1 << 24:
            tried.append(size)
        elif fake.is_counters(name, size):
            fake.counter(ptr, PATHS_DONE).value = 1 << 40

    with fake.on(see):
        r.autotune(spp=1, max_depth=2)
    assert len(tried) >= 2  # twice and four times the paths
    r.close(), scene.close()


def test_a_size_that_fits_only_unrounded(fake):
    """Sizes are rounded up to make kept blocks useful again, not at the price of an allocation that fits."""
    api = fake.api
    scene = api.Scene(api.Context(0), DESC)
    paths, more = 2_000_000, 2_020_000  # 264 bytes each: 528 and 533 MB, both rounded up to 537
    asked = []

    def see(name, ptr, size, stream):
        if name == "cudaMalloc" and size > 1 << 28:
            asked.append(size)

    fake.lib.fake_set_capacity(fake.lib.fake_allocated() + 264 * paths + (2 << 20))
    api.Renderer(scene, 64, 64, pool_size=paths).close()
    fake.lib.fake_set_capacity(180 << 30)
    with fake.on(see):
        api.Renderer(scene, 64, 64, pool_size=more).close()
    assert asked and asked[0] >= 264 * more  # not the smaller block
    scene.close()


def test_host_memory_runs_out_while_a_block_is_kept(fake):
    """A handle's destruction reports nothing, so it may not throw either (in a process of its own: it would abort)."""
    code = f"""
import sys
from pathlib import Path
sys.path[:0] = [{str(Path(__file__).parent)!r}, {str(Path(__file__).parent.parent)!r}]
from host_runtime import FakeRuntime
from test_kept_memory import DESC
rt = FakeRuntime(Path({str(fake.path)!r}))
scene = rt.api.Scene(rt.api.Context(0), DESC)
before = rt.lib.fake_allocated()
r = rt.api.Renderer(scene, 64, 64, pool_size=1 << 20)
rt.lib.fake_fail_new(100)
rt.lib.rmd_renderer_destroy(r.h)
rt.lib.fake_fail_new(0)
r.h = type(r.h)()
assert rt.lib.fake_allocated() == before, (rt.lib.fake_allocated(), before)  # freed, as nothing could be kept
rt.api.Renderer(scene, 64, 64, pool_size=1 << 20).close()
scene.close()
print("done")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("kind", ["renderer", "batch"])
def test_a_guide_that_ran_out_of_memory_is_set_up_whole(fake, kind):
    """Wherever set_guide runs out of memory, the next call allocates what is missing: no kernel gets a null buffer."""
    api = fake.api

    def make():
        ctx = api.Context(0)  # nothing kept
        if kind == "batch":
            return api.Batch(ctx, [DESC], [{"scene": 0, "width": 8, "height": 8}], pool_size=1 << 12)
        return api.Renderer(api.Scene(ctx, DESC), 8, 8, pool_size=1 << 12)

    def set_guide(x, fail_from):
        calls = 0

        def see(name, ptr, size, stream):
            nonlocal calls
            if name == "cudaMalloc":
                calls += 1
                return OUT_OF_MEMORY if fail_from <= calls else 0

        with fake.on(see):
            x.set_guide(sampling=True, training=True, replay_records=1 << 12)
        return calls

    def begin():
        x = make()
        with pytest.raises(api.RmdError, match="OUT_OF_MEMORY"):
            set_guide(x, 1)  # gives back what the context keeps
        return x, fake.lib.fake_allocated()

    x, base = begin()
    calls = set_guide(x, 1000)
    whole = fake.lib.fake_allocated() - base
    x.close()
    del x  # with its scene and context
    assert calls >= 16
    for k in range(1, calls + 1):
        x, base = begin()
        with pytest.raises(api.RmdError, match="OUT_OF_MEMORY"):
            set_guide(x, k)
        set_guide(x, 1000)
        assert fake.lib.fake_allocated() - base == whole, k
        x.close()
        del x
