"""Timed renders: every stage's kernels under their own names, and nothing else in the times."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    return compile_with_oracle(b.scene), compile_camera(b.camera), trace_settings({"global_illumination": True,
                                                                                   "max_bounces": 3})


@pytest.fixture
def gpu():
    from meercadraytracer_b200.executors import GpuExecutor

    ex = GpuExecutor(0)
    yield ex
    ex.dispose()


@pytest.mark.parametrize("size", [(64, 48), (320, 240)])  # few paths from the start, and at the end
def test_every_stage_is_counted(small, gpu, size):
    w, h = size
    want = gpu.raytrace(*small[:2], w, h, small[2], 2, True)
    plain = gpu.stats()
    gpu.set_timing(True)
    gpu.reset_stats()
    got = gpu.raytrace(*small[:2], w, h, small[2], 2, True)
    s = gpu.stats()
    assert np.array_equal(got, want)
    for key in ("closest_rays", "any_rays", "samples"):
        assert s[key] == plain[key]
    # One bounce more than may continue at most, each with a walk, a shading step and a resolve.
    assert 3 <= s["n_extend"] == s["n_shade"] == s["n_resolve"] and 1 <= s["n_shadow"] <= s["n_extend"]
    assert s["ms_shade"] > 0 and s["ms_shadow"] > 0 and s["ms_resolve"] > 0


def test_the_images_copy_is_in_no_stage(small, gpu):
    n = 2048
    gpu.set_timing(True)
    best = float("inf")
    for _ in range(3):
        gpu.reset_stats()
        gpu.raytrace(*small[:2], n, n, small[2], 1, True)
        best = min(best, gpu.stats()["ms_accumulate"])
    # The image alone, at the most a PCIe 5.0 x16 link carries.
    assert best < n * n * 4 / 64e9 * 1e3
