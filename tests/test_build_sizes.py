"""The two-phase builder at the edges of its phases and sizes: the oracle's tree, numbered breadth first.

Nodes of more than 256 triangles are split level by level in segments of 512 to
4,096 triangles, smaller ones are finished in shared memory, leaves hold up to
4 (16 when splitting costs more). The sizes straddle each of these; the last
case is a chain whose large nodes go far deeper than a balanced tree's, so the
level loop has to be extended.
"""
import numpy as np
import pytest

from oracle import cpu
from test_full_size import canonical
from test_oracle_bvh_color import lcg_triangles

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


def check(gpu, raw, n):
    ob, oo = cpu.build_bvh(raw, n)
    gb, go = gpu.build_bvh(raw, n)
    assert np.array_equal(np.sort(go), np.arange(n))
    assert gb.node_count == ob.node_count
    assert canonical(gb, go) == canonical(ob, oo)
    assert sorted(map(tuple, gb.bounds.reshape(-1, 6).tolist())) == sorted(map(tuple, ob.bounds.reshape(-1, 6).tolist()))
    # Breadth first: the k-th inner node's children are nodes 1 + 2k and 2 + 2k.
    nodes = gb.nodes.reshape(-1, 3)
    inner = nodes[nodes[:, 1] == 0]
    assert np.array_equal(inner[:, 0], 1 + 2 * np.arange(inner.shape[0]))
    # Leaves tile the triangles.
    leaves = nodes[nodes[:, 1] > 0]
    leaves = leaves[np.argsort(leaves[:, 0])]
    assert np.array_equal(np.cumsum(leaves[:, 1])[:-1], leaves[1:, 0]) and leaves[:, 1].sum() == n


@pytest.mark.parametrize("n", [1, 2, 4, 5, 15, 16, 17, 31, 32, 33, 64, 65, 255, 256, 257, 511, 512, 513, 1023, 1025,
                               4095, 4097, 8193, 60_001])
def test_sizes_match_the_oracle(gpu, n):
    check(gpu, lcg_triangles(n, 100 + n), n)


def test_smaller_build_after_a_larger_one(gpu):
    for n in (20_000, 300, 20_000, 7, 3_000):
        check(gpu, lcg_triangles(n, n), n)


def test_chain_of_large_nodes_matches_the_oracle(gpu):
    n = 1200
    x = 1e-20 * 1.07 ** np.arange(n)
    raw = np.zeros((n, 9), np.float32)
    raw[:, 0] = x
    raw[:, 3] = raw[:, 7] = 0.01 * x
    check(gpu, raw.reshape(-1), n)
