"""The pool's memory goes back when the last executor or batch is disposed, and the rest when it is dropped."""
import gc

import numpy as np
import pytest

from meercadraytracer_b200 import pinned
from test_host_memory import HostPool


def test_free_blocks_go_with_the_last_user(monkeypatch):
    pool = HostPool(monkeypatch)
    pool.attach()
    pool.attach()
    for _ in range(4):
        pool.empty(1 << 20, np.uint8)
        pool.empty(1 << 22, np.uint8)
    gc.collect()
    assert pool.blocks
    pool.detach()
    assert pool.blocks
    pool.detach()
    assert not pool.blocks and pool._held == 0


def test_a_kept_result_goes_when_it_is_dropped(monkeypatch):
    pool = HostPool(monkeypatch)
    pool.attach()
    kept = pool.empty(1 << 20, np.uint8)
    kept[:] = 7
    pool.detach()
    assert len(pool.blocks) == 1 and (kept == 7).all()
    del kept
    gc.collect()
    assert not pool.blocks and pool._held == 0


@pytest.mark.parametrize("kept", [False, True])
def test_the_pool_serves_the_next_user(monkeypatch, kept):
    pool = HostPool(monkeypatch)
    pool.attach()
    first = pool.empty(1 << 20, np.uint8)
    pool.detach()
    if not kept:
        del first
    pool.attach()
    results = [pool.empty(1 << 20, np.uint8) for _ in range(2)]
    assert all(a.base is not None for a in results)
    address = results[0].ctypes.data
    del results
    gc.collect()
    again = [pool.empty(1 << 20, np.uint8) for _ in range(2)]  # blocks are kept for reuse again
    assert address in [a.ctypes.data for a in again]


@pytest.mark.gpu
def test_executors_and_batches_return_it():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.batch import BatchRenderer, RenderRequest
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.executors import GpuExecutor
    from meercadraytracer_b200.raytrace import trace_settings

    gc.collect()
    before = pinned._pool.users
    b = scenes.small_scene()
    compiled, cam, st = compile_with_oracle(b.scene), compile_camera(b.camera), trace_settings({})
    ex, batch = GpuExecutor(0), BatchRenderer(0, capacity=1 << 18, memory_budget=64 << 20)
    ex.raytrace(compiled, cam, 320, 240, st, 1, True)
    batch.adopt(compiled, ex)
    (image,) = batch.render([RenderRequest(compiled, cam, 320, 240, st, 1)])
    want = image.copy()
    batch.dispose()
    ex.dispose()
    ex.dispose()  # once is enough
    assert pinned._pool.users == before
    if before == 0:
        assert not any(pinned._pool._free.values())
    assert np.array_equal(image, want)
