"""Results in pinned memory: blocks are reused only when nothing refers to them, and the pool is bounded."""
import gc

import numpy as np
import pytest

from meercadraytracer_b200 import pinned
from meercadraytracer_b200.pinned import _Pool


class HostPool(_Pool):
    """The pool over a stand-in for the driver's allocator (ctypes memory)."""

    def __init__(self, monkeypatch, fail=False):
        super().__init__()
        import ctypes as C

        self.blocks = {}

        def call(name, *args):
            if name == "mcrt_host_alloc":
                if fail:
                    raise pinned.McrtError(2, "no memory")
                block = (C.c_uint8 * args[0])()
                self.blocks[C.addressof(block)] = block
                args[1]._obj.value = C.addressof(block)
            else:
                del self.blocks[args[0].value]

        monkeypatch.setattr(pinned, "call", call)


def test_blocks_return_with_their_last_view(monkeypatch):
    pool = HostPool(monkeypatch)
    a = pool.empty(100_000, np.float32)
    address = a.ctypes.data
    view = a[10:20]
    del a
    gc.collect()
    b = pool.empty(100_000, np.float32)  # the view holds the first block
    assert b.ctypes.data != address
    del view
    gc.collect()
    c = pool.empty(100_000, np.float32)
    assert c.ctypes.data == address and len(pool.blocks) == 2
    assert b.flags.writeable and b.dtype == np.float32 and b.shape == (100_000,)


def test_small_arrays_and_a_full_pool_are_ordinary_memory(monkeypatch):
    monkeypatch.setattr(pinned, "LIMIT", 1 << 20)
    pool = HostPool(monkeypatch)
    assert pool.empty(10, np.uint8).base is None and not pool.blocks
    held = [pool.empty(1 << 19, np.uint8) for _ in range(3)]
    assert len(pool.blocks) == 2 and held[2].base is None
    assert pool.empty(1 << 21, np.uint8).base is None
    held.clear()
    gc.collect()
    big = pool.empty(1 << 20, np.uint8)  # the free blocks of another size make room
    assert big.base is not None and len(pool.blocks) == 1


def test_an_allocation_failure_is_ordinary_memory(monkeypatch):
    pool = HostPool(monkeypatch, fail=True)
    assert pool.empty(1 << 20, np.uint8).base is None
    assert pool._held == 0


def test_size_classes_waste_little():
    for n in (1 << 16, 100_001, 8_294_400, (1 << 27) + 1):
        size = _Pool.block_size(n)
        assert n <= size <= n * 1.25 + 4096 and _Pool.block_size(size) == size


@pytest.mark.gpu
def test_held_images_keep_their_pixels():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.executors import GpuExecutor
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    compiled, cam = compile_with_oracle(b.scene), compile_camera(b.camera)
    ex = GpuExecutor(0)
    try:
        images = [ex.raytrace(compiled, cam, 200, 150, trace_settings({"seed": s}), 1 + s) for s in range(4)]
        again = [ex.raytrace(compiled, cam, 200, 150, trace_settings({"seed": s}), 1 + s) for s in range(4)]
        assert all(np.array_equal(x, y) for x, y in zip(images, again))
        assert len({x.ctypes.data for x in images + again}) == 8
    finally:
        ex.dispose()


@pytest.mark.gpu
def test_a_cancelled_requests_buffers_outlive_its_copies():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.batch import BatchRenderer, RenderRequest
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    compiled, cam = compile_with_oracle(b.scene), compile_camera(b.camera)
    r = BatchRenderer(0, capacity=1 << 18, memory_budget=64 << 20)
    try:
        rid = r.submit(RenderRequest(compiled, cam, 320, 240, trace_settings({}), 8, 4, progress=True))
        r.step()
        r.cancel(rid)
        r.forget(rid)
        assert len(r._retired) == 1
        for _ in range(3):
            r.step()
        assert not r._retired
    finally:
        r.dispose()
