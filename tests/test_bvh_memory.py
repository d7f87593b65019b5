"""A hierarchy holds the memory of its own nodes, not of the most that its triangles could make."""
import numpy as np
import pytest

from meercadraytracer_b200._lib import McrtError, call
from test_oracle_bvh_color import lcg_triangles

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


def held(a):
    """Bytes that stay allocated while `a` does."""
    while isinstance(a.base, np.ndarray):
        a = a.base
    return a.nbytes


@pytest.mark.parametrize("n", [0, 1, 5, 700, 20_000])
def test_arrays_have_the_hierarchys_size(gpu, n):
    bvh, order = gpu.build_bvh(lcg_triangles(max(n, 1), 3)[: 9 * n], n)
    assert bvh.bounds.size == held(bvh.bounds) // 4 == 6 * bvh.node_count
    assert bvh.nodes.size == held(bvh.nodes) // 4 == 3 * bvh.node_count
    assert order.size == held(order) // 4 == n
    assert np.array_equal(np.sort(order), np.arange(n))


def test_there_is_nothing_to_read_after_another_compile(gpu):
    import ctypes as C

    from helpers import floor
    from meercadraytracer_b200 import scene as S
    from meercadraytracer_b200.compile import compile_scene

    gpu.build_bvh(lcg_triangles(9, 3), 9)
    scene = S.Scene()
    scene.add(floor(S.MeshBasicMaterial()))
    compile_scene(scene, builder=gpu.compile_sink)
    out = (C.c_float * 600)(), (C.c_int32 * 300)(), (C.c_uint32 * 100)()
    with pytest.raises(McrtError):
        call("mcrt_bvh_read", gpu._h, *out)
