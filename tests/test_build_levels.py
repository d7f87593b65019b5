"""Level kernels in smaller blocks: the oracle's tree at the sizes where the block size changes.

A level with four segments per SM (592 of 512 triangles) is split by blocks of
128 threads, one with eight (1184) by blocks of 64; below, by 256. Sizes stand
on both sides of each, with triangles spread evenly (balanced trees) and
clustered (large nodes far down, and bins that take most of a node).
"""
import numpy as np
import pytest

from test_build_sizes import check
from test_oracle_bvh_color import lcg_triangles

pytestmark = pytest.mark.gpu

FOUR, EIGHT = 592 * 512, 1184 * 512


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


@pytest.mark.parametrize("n", [FOUR - 1, FOUR, EIGHT - 1, EIGHT + 300])
def test_even_triangles(gpu, n):
    check(gpu, lcg_triangles(n, n % 1000), n)


@pytest.mark.parametrize("n", [FOUR + 511, EIGHT])
def test_clustered_triangles(gpu, n):
    rng = np.random.default_rng(n)
    centre = rng.normal(size=(n, 3)) * 10.0 ** rng.integers(-4, 3, size=(n, 1))
    raw = np.repeat(centre, 3, axis=0).reshape(n, 9) + rng.normal(size=(n, 9)) * 1e-3
    check(gpu, raw.astype(np.float32).reshape(-1), n)
