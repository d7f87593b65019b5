"""Camera rays of many paths: the same samples as of few.

A chunk of at least 65536 paths is shaded in class order: its first walk knows
queue and flags without reading them and gives misses under a background of one
colour their sample itself; where the rays are coherent it makes them too.
Fewer paths take the queued stages, and up to 8192 one launch. Running sums must
agree bit for bit with those of calls for few pixels, over every kind of
background, cut-outs, fog and tone map of the random scenes. The coherent walk
may take the other of two hits at exactly equal distance: there at most one
pixel in 500 may differ.
"""
import numpy as np
import pytest

from test_random_scenes import H, W, _prepare

pytestmark = pytest.mark.gpu

FEW = 8192      # paths that one launch finishes
SORT = 1 << 16  # paths shaded in class order
TALL = 720      # image height at which 16 or more passes of a pixel walk coherently


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


def few_at_a_time(gpu, compiled, cam, w, h, st, spp, srgb, px, py):
    step = FEW // spp
    parts = [gpu.render_pixels(compiled, cam, w, h, st, spp, srgb, px[i:i + step], py[i:i + step])
             for i in range(0, px.size, step)]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


@pytest.mark.parametrize("gi", [False, True])
@pytest.mark.parametrize("seed", range(12))
def test_sorted_start(gpu, seed, gi):
    compiled, cam, st, spp, srgb, px, py = _prepare(seed)
    st.global_illumination = gi
    rgba, sums = few_at_a_time(gpu, compiled, cam, W, H, st, 1, srgb, px, py)
    repeat = SORT // px.size + 1
    many_rgba, many = gpu.render_pixels(compiled, cam, W, H, st, 1, srgb, np.tile(px, repeat), np.tile(py, repeat))
    assert np.array_equal(many.reshape((repeat,) + sums.shape), np.broadcast_to(sums, (repeat,) + sums.shape))
    assert np.array_equal(many_rgba.reshape((repeat,) + rgba.shape), np.broadcast_to(rgba, (repeat,) + rgba.shape))


@pytest.mark.parametrize("n", [FEW + 1, SORT - 1, SORT, SORT + 1, SORT + 127])
def test_path_counts(gpu, n):
    compiled, cam, st, spp, srgb, px, py = _prepare(3)
    at = (np.arange(n) * 13 + 5) % px.size
    _, base = few_at_a_time(gpu, compiled, cam, W, H, st, 1, srgb, px, py)
    _, sums = gpu.render_pixels(compiled, cam, W, H, st, 1, srgb, px[at], py[at])
    assert np.array_equal(sums, base[at])


@pytest.mark.parametrize("pixels", [400, 4097])  # below and above the sorted start at 16 passes
@pytest.mark.parametrize("seed", range(6))
def test_coherent_start(gpu, seed, pixels):
    compiled, cam, st, _, srgb, _, _ = _prepare(seed)
    rng = np.random.default_rng(seed)
    w, spp = TALL * W // H, 24
    x0, y0 = int(rng.integers(w // 4, w // 2)), int(rng.integers(TALL // 4, TALL // 2))
    i = np.arange(pixels)
    px, py = (x0 + i % 64).astype(np.int32), (y0 + i // 64).astype(np.int32)
    assert pixels * spp > FEW
    _, want = few_at_a_time(gpu, compiled, cam, w, TALL, st, spp, srgb, px, py)
    _, got = gpu.render_pixels(compiled, cam, w, TALL, st, spp, srgb, px, py)
    differ = np.any(want != got, axis=-1).reshape(-1)
    assert np.count_nonzero(differ) * 500 <= pixels
