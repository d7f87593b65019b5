"""A shadow ray that is blocked on the last step of its budget has its answer: no limit was reached.

A floor under four roofs, the camera between floor and lowest roof, the light
above all: floor and lowest roof share a leaf, so a camera ray takes the root
and that leaf, and a shadow ray is blocked there while the upper roofs wait.
"""
import numpy as np
import pytest

from meercadraytracer_b200 import scene as S
from meercadraytracer_b200._lib import McrtError

pytestmark = pytest.mark.gpu


def roofs():
    scene = S.Scene()
    for z in range(5):
        mesh = S.Mesh(S.plane_geometry(4, 4), S.MeshLambertMaterial(color=0xffffff, side=S.DoubleSide))
        mesh.position.set(0, 0, z)
        scene.add(mesh)
    light = S.DirectionalLight(0xffffff, 2.0)
    light.position.set(0, 0, 10)
    scene.add(light, S.AmbientLight(0xffffff, 0.5))
    camera = S.OrthographicCamera(-1, 1, 1, -1, 0.1, 100)
    camera.position.set(0, 0, 0.5)
    camera.look_at(0, 0, 0)
    camera.update_matrix_world()
    return scene, camera


@pytest.mark.parametrize("size", [16, 128])  # one launch for all paths, and the wavefront's queues
def test_blocked_on_the_last_step(size):
    from helpers import compile_with_oracle
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.executors import GpuExecutor
    from meercadraytracer_b200.raytrace import trace_settings

    scene, camera = roofs()
    compiled, cam, st = compile_with_oracle(scene), compile_camera(camera), trace_settings({})
    bvh = compiled.geometry.bvh.nodes.reshape(-1, 3)
    assert bvh[0, 1] == 0 and 4 in bvh[bvh[0, 0]:bvh[0, 0] + 2, 1]
    ex = GpuExecutor(0)
    try:
        want = ex.raytrace(compiled, cam, size, size, st, 1, True)
        ex.set_step_limit(2)
        assert np.array_equal(ex.raytrace(compiled, cam, size, size, st, 1, True), want)
        ex.set_step_limit(1)
        with pytest.raises(McrtError):
            ex.raytrace(compiled, cam, size, size, st, 1, True)
    finally:
        ex.dispose()
