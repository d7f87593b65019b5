"""Result memory is allocated from the device whose results it takes, not from whichever a thread starts on."""
import ctypes as C
import threading

import numpy as np
import pytest

from meercadraytracer_b200 import batch, executors, pinned
from meercadraytracer_b200.types import Tile
from test_batch_buffers import Scene, engine  # noqa: F401 (fixture)


@pytest.mark.parametrize("device", [0, 3])
def test_new_blocks_come_from_the_device(monkeypatch, device):
    calls = []

    def call(name, *args):
        calls.append((name, args[0]))
        raise pinned.McrtError(2, "no memory")

    monkeypatch.setattr(pinned, "call", call)
    pinned._Pool().empty(1 << 20, np.uint8, device)
    assert calls == [("mcrt_host_alloc_on", device)]


@pytest.fixture
def devices(monkeypatch):
    """The devices that results are asked for, of executors and batches without a library."""
    seen = []
    for name in ("empty", "zeros"):
        monkeypatch.setattr(pinned, name, lambda n, dtype, device=None: (seen.append(device), np.zeros(n, dtype))[1])
    monkeypatch.setattr(executors, "call", lambda *a: None)
    return seen


def test_executors_name_their_device(devices, monkeypatch):
    for name in ("to_c_camera", "to_c_settings", "to_c_tile"):
        monkeypatch.setattr(executors.abi, name, lambda v: C.c_int())
    ex = executors.GpuExecutor.__new__(executors.GpuExecutor)
    ex._disposed, ex._h, ex._lock, ex.device = True, C.c_void_p(1), threading.Lock(), 2
    ex._geometry_version = ex._shading_version = 1
    ex._render_tile({"tile": Tile(0, 0, 8, 8), "camera": None, "settings": None, "geometry_version": 1,
                     "shading_version": 1, "width": 8, "height": 8, "pass": 0, "block": 1})
    ex.raytrace_resident((1, 1), None, 8, 8, None, 1)
    ex.intersect_closest(1, np.zeros((4, 8), np.float32))
    ex.intersect_any_count(1, np.zeros((4, 8), np.float32))
    ex.build_bvh(np.zeros(9, np.float32), 1)
    assert devices and set(devices) == {2}


def test_batches_name_their_device(devices, engine):  # noqa: F811
    r = batch.BatchRenderer(device=2)
    r.submit_to(Scene(), (1, 1), None, None, 8, 8, 4, preview_block=4, progress=True)
    assert devices == [2, 2, 2]
