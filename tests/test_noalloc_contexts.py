"""Contexts made while rmd_render_noalloc renders."""
import threading
import time

import numpy as np
import pytest

from host_runtime import PATHS_DONE, fake  # noqa: F401
from raymond_b200 import scenes
from raymond_b200._abi import SceneDesc

W, H = 64, 48


def test_a_running_call_keeps_its_events(fake):
    """A context made while a call's work is pending (on the host, the device's part played by the test): the call goes on
    with the events it began with."""
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    scene = api.Scene(api.Context(0), desc)
    film = np.zeros((H, W, 4), np.float32)
    others, recorded, waited = [], [], []
    reads = 0

    def see(name, ptr, size, stream):
        nonlocal reads
        if fake.is_counters(name, size):
            reads += 1
            if reads == 4:  # the paths have ended
                fake.counter(ptr, PATHS_DONE).value = W * H
        elif name == "cudaEventRecord":
            recorded.append(ptr)
            if len(recorded) in (1, 2):  # pending now
                others.append(api.Context(0))
        elif name == "cudaEventSynchronize":
            waited.append(ptr)

    with fake.on(see):
        api.render_noalloc(scene, desc.scene["camera"], W, H, film.ctypes.data, spp=1, first_sample=0, max_depth=4)
    assert reads >= 4 and len(set(recorded)) == 2  # two events in turn
    assert waited == recorded[:len(waited)]


def test_a_context_after_a_device_reset(fake):
    """What went with a device reset is not used by a context made after it (a stale handle is undefined behaviour)."""
    api = fake.api
    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=2))
    film = np.zeros((H, W, 4), np.float32)

    def see(name, ptr, size, stream):
        if fake.is_counters(name, size):
            fake.counter(ptr, PATHS_DONE).value = W * H

    for _ in range(2):
        scene = api.Scene(api.Context(0), desc)
        with fake.on(see):
            api.render_noalloc(scene, desc.scene["camera"], W, H, film.ctypes.data, spp=1, first_sample=0, max_depth=4)
        fake.lib.fake_reset_device()
    assert fake.lib.fake_stale_uses() == 0


@pytest.mark.gpu
def test_contexts_beside_a_render(gpu_ctx):
    """Contexts created and dropped on another thread while noalloc renders run: every film is the one rendered alone."""
    import torch

    from raymond_b200 import api

    desc = SceneDesc(scenes.cornell(seed=1, envmap_exponent=6))
    scene = api.Scene(gpu_ctx, desc)
    film = torch.zeros((H, W, 4), device="cuda")

    def render():
        film.zero_()
        torch.cuda.synchronize()
        api.render_noalloc(scene, desc.scene["camera"], W, H, film.data_ptr(), spp=1, first_sample=0, max_depth=8)
        return film.cpu().numpy()

    alone = render()
    stop, failed, made = threading.Event(), [], [0]

    def contexts():
        try:
            while not stop.is_set():
                api.Context(0).close()
                made[0] += 1
        except Exception as e:  # reported by the main thread
            failed.append(e)

    t = threading.Thread(target=contexts)
    t.start()
    try:
        films, until = [], time.monotonic() + 60
        while (len(films) < 300 or made[0] < 20) and not failed and time.monotonic() < until:
            films.append(render())
    finally:
        stop.set()
        t.join()
    assert not failed and made[0] > 10
    for f in films:
        np.testing.assert_array_equal(f, alone)
