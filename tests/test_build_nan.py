"""Triangles with NaN vertices do not spoil the hierarchy of the others: the oracle's tree."""
import numpy as np
import pytest

from test_build_sizes import check
from test_oracle_bvh_color import lcg_triangles

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


@pytest.mark.parametrize("axes", [[0, 1, 2], [0], [2]])
@pytest.mark.parametrize("n", [9, 14, 40, 255, 700, 5000, 30_001])
def test_nan_vertices_match_the_oracle(gpu, n, axes):
    raw = lcg_triangles(n, 7 + n).reshape(-1, 9).copy()
    for t in {0, n // 3, n - 1}:
        raw[t, axes] = np.nan
    check(gpu, raw.reshape(-1), n)
