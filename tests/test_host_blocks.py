"""mcrt_host_alloc: blocks of every size apart from one another, from any thread, and a forked child's own copy."""
import ctypes as C
import gc
import os
import signal
import threading

import numpy as np
import pytest

from meercadraytracer_b200._lib import McrtError, call

pytestmark = pytest.mark.gpu

MB = 1 << 20
SIZES = [1, 4096, 4097, 65536, 100_000, MB, 2 * MB - 4096, 2 * MB, 2 * MB + 1, 4 * MB, 4 * MB + 4096, 9 * MB + 5]


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


def alloc(size):
    p = C.c_void_p()
    call("mcrt_host_alloc_on", 0, size, C.byref(p))
    assert p.value % 4096 == 0
    return np.frombuffer((C.c_uint8 * size).from_address(p.value), np.uint8)


def free(a):
    call("mcrt_host_free", C.c_void_p(a.ctypes.data))


def test_blocks_do_not_overlap(gpu):
    rng = np.random.default_rng(1)
    held = []
    for step in range(300):
        if held and rng.random() < 0.45:
            a, v = held.pop(int(rng.integers(len(held))))
            assert (a == v).all()
            free(a)
        else:
            a, v = alloc(int(rng.choice(SIZES))), step % 251 + 1
            a[:] = v
            held.append((a, v))
    for a, v in held:
        assert (a == v).all()
        free(a)


def test_a_block_is_freed_once_and_no_size_is_too_large_to_refuse(gpu):
    for size in SIZES:
        a = alloc(size)
        free(a)
        with pytest.raises(McrtError):
            free(a)
    for size in (1 << 50, (1 << 64) - 1):
        with pytest.raises(McrtError):
            alloc(size)


def test_other_threads_free_and_allocate(gpu):
    blocks, errors = [alloc(s) for s in SIZES for _ in range(4)], []

    def work(mine):
        try:
            for a in mine:
                free(a)
            for s in SIZES:
                free(alloc(s))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(blocks[i::4],)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_a_forked_child_keeps_its_image(gpu):
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    compiled, cam = compile_with_oracle(b.scene), compile_camera(b.camera)
    image = gpu.raytrace(compiled, cam, 320, 240, trace_settings({"seed": 1}), 1, True)
    assert image.base is not None  # pinned
    want, at = image.copy(), image.ctypes.data
    ready, go = os.pipe(), os.pipe()
    gc.collect()
    gc.disable()  # no finalizer, and so no CUDA call, runs in the child
    try:
        child = os.fork()
        if child == 0:  # memory only
            signal.alarm(60)
            os.write(ready[1], b"x")
            os.read(go[0], 1)
            os._exit(0 if np.array_equal(image, want) else 1)
    finally:
        gc.enable()
    os.read(ready[0], 1)
    del image
    later = gpu.raytrace(compiled, cam, 320, 240, trace_settings({"seed": 2}), 1, True)
    assert later.ctypes.data == at and not np.array_equal(later, want)
    os.write(go[1], b"x")
    assert os.waitstatus_to_exitcode(os.waitpid(child, 0)[1]) == 0
