"""Instances as compile_instances takes them: rows of six, integers narrowed to the fields' widths."""
import ctypes as C
import threading

import numpy as np
import pytest

from meercadraytracer_b200 import executors

ROW = (np.eye(4), 0, 1, 1, 0, False)


@pytest.fixture
def compiled(monkeypatch):
    """compile_instances up to the library call; the list receives the C structs."""
    seen = []

    def call(name, *args):
        assert name == "mcrt_compile_instances"
        seen.extend(args[3][:args[2]])

    monkeypatch.setattr(executors, "call", call)
    ex = executors.GpuExecutor.__new__(executors.GpuExecutor)
    ex._disposed, ex._h, ex._lock, ex._versions = True, C.c_void_p(1), threading.Lock(), 0
    return lambda rows: (ex.compile_instances(rows), seen)[1]


@pytest.mark.parametrize("rows", [[ROW + (0,), ROW], [ROW, ROW + (0,)], [ROW[:5]], [ROW + (0,)], [ROW, ROW[:5]]])
def test_rows_of_another_length_are_refused(compiled, rows):
    with pytest.raises(ValueError):
        compiled(rows)


@pytest.mark.parametrize("value", [0, -1, 255, 256, (1 << 32) - 1, (1 << 63) + 5, 1 << 64, -(1 << 70) + 3, np.uint64(1 << 63)])
def test_integers_keep_their_low_bits(compiled, value):
    (c,) = compiled([(np.eye(4), value, value, value, value, False)])
    assert c.mesh == C.c_int32(int(value)).value and c.material == C.c_uint32(int(value)).value
    assert c.flags == C.c_uint8(int(value)).value and c.side == C.c_uint8(int(value)).value
