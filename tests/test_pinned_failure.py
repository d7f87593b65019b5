"""Pinned memory that is not to be had: the caller goes on in ordinary memory."""
import ctypes as C

import numpy as np
import pytest

from meercadraytracer_b200._lib import McrtError, call

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_does_not_fail_the_next_call():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.executors import GpuExecutor
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    compiled, cam, st = compile_with_oracle(b.scene), compile_camera(b.camera), trace_settings({})
    ex = GpuExecutor(0)
    try:
        want = ex.raytrace(compiled, cam, 64, 48, st, 1, True)
        p = C.c_void_p()
        with pytest.raises(McrtError):
            call("mcrt_host_alloc", 1 << 50, C.byref(p))
        assert not p.value
        assert np.array_equal(ex.raytrace(compiled, cam, 64, 48, st, 1, True), want)
    finally:
        ex.dispose()
