"""Reading results back: sizes below and above the pinned path's limit, odd ones, two sessions read from two threads at
once (one of them finds the pinned slots taken), and destinations that are pinned memory themselves."""
import threading
import time

import numpy as np
import pytest
import torch

from rtcuda import PtSession, abi, backend, scenes

pytestmark = pytest.mark.gpu


def _check(g):
    acc, img, aux, film = g.sum_and_weight(), g.image(), g.aux(), g.film_array()
    assert np.array_equal(img, (acc[..., :3] / acc[..., 3:]).astype(np.float32))
    assert np.array_equal(film[..., 0:3], img)
    hits = aux[..., 11]
    assert np.array_equal(film[..., 16], aux[..., 7]) and (hits <= acc[..., 3]).all()
    assert (acc[..., 3] == acc[0, 0, 3]).all()


@pytest.mark.parametrize("w,h", [(64, 48), (591, 592), (1031, 1021), (1920, 1080)])
def test_layers_agree(w, h):
    with PtSession(scenes.cornell_box(w, h), abi.make_params(max_depth=2, aovs=True)) as g:
        g.render_samples(0, 1)
        _check(g)
        g.render_samples(1, 2)
        _check(g)


def test_two_threads():
    errors = []

    def work(k):
        try:
            with PtSession(scenes.cornell_box(1300 + k, 900), abi.make_params(max_depth=2, aovs=True)) as g:
                g.render_samples(k, 1)
                for _ in range(6):
                    _check(g)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    t = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not errors, errors


def _best(f):
    times = []
    for _ in range(8):
        t = time.perf_counter()
        f()
        times.append(time.perf_counter() - t)
    return min(times)


def test_pinned_destinations_are_written_directly():
    """A result read into pinned memory takes one copy, not a second one through the slots: about the time of that copy
    (through the slots it took half as long again or twice as long)."""
    lib = backend.lib()
    with PtSession(scenes.cornell_box(1920, 1080), abi.make_params(max_depth=2, aovs=True)) as g:
        g.render_samples(0, 1)
        want = g.film_array()
        pinned = torch.full((1080, 1920, 18), -1.0, pin_memory=True)
        read = _best(lambda: backend._check(lib.rt_read_film(g.h, pinned.data_ptr())))
        assert np.array_equal(pinned.numpy(), want)
        device = torch.zeros((1080, 1920, 18), device="cuda")
        copy = _best(lambda: (pinned.copy_(device, non_blocking=True), torch.cuda.synchronize()))
    assert read < 1.25 * copy + 4e-4, (read, copy)   # the film is decoded on the device first


def test_release_memory_gives_back_and_leaves_sessions_usable():
    """What destroyed sessions returned to the pool goes back to the driver; the pinned slots are made anew."""
    keep = PtSession(scenes.cornell_box(64, 48), abi.make_params(max_depth=2, aovs=True))
    with PtSession(scenes.cornell_box(1300, 900), abi.make_params(max_depth=2, aovs=True)) as g:
        g.render_samples(0, 1)
        _check(g)
        held = g.stats()["device_bytes"]
    free = torch.cuda.mem_get_info()[0]
    backend.release_memory()
    assert torch.cuda.mem_get_info()[0] - free > 0.5 * held > 1 << 20
    backend.release_memory()
    keep.render_samples(0, 1)
    _check(keep)
    keep.close()
    with PtSession(scenes.cornell_box(1300, 900), abi.make_params(max_depth=2, aovs=True)) as g:
        g.render_samples(0, 1)
        _check(g)
