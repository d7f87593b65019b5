"""Queues of few paths are taken to their ends in one launch: the same samples as bounce by bounce.

A call for few pixels runs whole in that launch; the same pixels inside a call
for many run through the wavefront's queues until few paths are left. Running
sums must agree bit for bit (every stage's arithmetic is the same), the counted
queries must be the same per path, and the batch engine's images must equal the
plain path's. Scenes cover every material model, maps, cut-outs, transparency,
every light type, shadow modes, fog, environments and tone maps.
"""
import numpy as np
import pytest

from test_random_scenes import H, W, _prepare

pytestmark = pytest.mark.gpu

FEW = 8192  # paths of a queue that one launch finishes


@pytest.fixture(scope="module")
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


def settings_of(st, gi):
    st.global_illumination = gi
    st.max_bounces = max(3, st.max_bounces)
    return st


@pytest.mark.parametrize("gi", [False, True])
@pytest.mark.parametrize("seed", range(12))
def test_few_paths_give_the_wavefronts_samples(gpu, seed, gi):
    compiled, cam, st, spp, srgb, px, py = _prepare(seed)
    st = settings_of(st, gi)
    repeat = 2 * FEW // (px.size * spp) + 2
    many_px, many_py = np.tile(px, repeat), np.tile(py, repeat)
    gpu.reset_stats()
    rgba, sums = gpu.render_pixels(compiled, cam, W, H, st, spp, srgb, many_px, many_py)
    many = gpu.stats()
    few = FEW // spp
    for first in range(0, px.size, few):
        part = slice(first, min(first + few, px.size))
        r, s = gpu.render_pixels(compiled, cam, W, H, st, spp, srgb, px[part], py[part])
        assert np.array_equal(s, sums[part])
        assert np.array_equal(r, rgba[part])
    total = gpu.stats()
    for key in ("closest_rays", "any_rays", "samples"):
        assert (total[key] - many[key]) * repeat == many[key], key


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 63, 65, 2367, 2369, 4737, FEW, FEW + 1])
def test_path_counts(gpu, n):
    compiled, cam, st, spp, srgb, px, py = _prepare(3)
    st = settings_of(st, True)
    at = (np.arange(n) * 13 + 5) % px.size
    base_rgba, base = gpu.render_pixels(compiled, cam, W, H, st, 1, srgb, np.tile(px, 9), np.tile(py, 9))
    assert 9 * px.size > FEW
    rgba, sums = gpu.render_pixels(compiled, cam, W, H, st, 1, srgb, px[at], py[at])
    assert np.array_equal(sums, base[at]) and np.array_equal(rgba, base_rgba[at])


def test_batched_images_equal_plain(gpu):
    from meercadraytracer_b200.batch import BatchRenderer, RenderRequest

    renderer = BatchRenderer(0, capacity=1 << 16, memory_budget=64 << 20)
    try:
        for seed in (0, 4, 7):
            compiled, cam, st, spp, srgb, _, _ = _prepare(seed)
            st = settings_of(st, True)
            want = gpu.raytrace(compiled, cam, W, H, st, 5, srgb)
            for preview in (0, 4):
                (got,) = renderer.render([RenderRequest(compiled, cam, W, H, st, 5, preview, srgb)])
                assert np.array_equal(got, want)
    finally:
        renderer.dispose()
