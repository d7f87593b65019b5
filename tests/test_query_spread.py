"""Few queries spread over many warps: a ray's answer does not depend on how many
rays its call has.

The walk gives each resident warp a power of two of a call's rays, from one
(fewer rays than warps) to 32 (the GPU is full), and refills warps from a
queue. Each call here repeats the same rays, whose answers the oracle checks,
at counts around those edges: one ray, a warp, one per warp of the smallest
and largest grids, and just past every power of two per warp.
"""
import numpy as np
import pytest

from helpers import compile_with_oracle
from meercadraytracer_b200 import scenes
from oracle import cpu

pytestmark = pytest.mark.gpu

RAYS = 97


@pytest.fixture(scope="module")
def setup():
    from meercadraytracer_b200.executors import GpuExecutor

    compiled = compile_with_oracle(scenes.small_scene().scene)
    ex = GpuExecutor(0)
    version, _ = ex.load_scene(compiled)
    rng = np.random.default_rng(5)
    rays = np.zeros((RAYS, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-8, 8, (RAYS, 3)) + (0, 9, 0)
    d = rng.normal(size=(RAYS, 3))
    d[:6] = np.concatenate([np.eye(3), -np.eye(3)])  # along every axis, both ways
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    yield ex, version, compiled.geometry, rays
    ex.dispose()


def test_oracle_agrees_on_the_repeated_rays(setup):
    ex, version, g, rays = setup
    hits = ex.intersect_closest(version, rays)
    for i in range(RAYS):
        found, h = cpu.intersect_closest(g.triangles, g.sides, g.bvh, rays[i, 0:3].astype(np.float64),
                                         rays[i, 4:7].astype(np.float64))
        assert found == (hits["tri"][i] >= 0)
        if found:
            assert abs(h.t - hits["t"][i]) <= 1e-5 * h.t


@pytest.mark.parametrize("n", [1, 2, 31, 33, 591, 593, 1024, 4095, 4096, 4097, 4735, 4737, 9473, 16383, 16384, 16385, 18945, 37889,
                               75777, 151553])
def test_answers_do_not_depend_on_the_number_of_rays(setup, n):
    ex, version, _, rays = setup
    base = ex.intersect_closest(version, rays)
    count = ex.intersect_any_count(version, rays)
    at = (np.arange(n) * 7 + n) % RAYS
    many = ex.intersect_closest(version, rays[at])
    for k in base:
        assert np.array_equal(many[k], base[k][at]), k
    assert np.array_equal(ex.intersect_any_count(version, rays[at]), count[at])
