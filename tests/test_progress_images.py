"""Images that a batch's events name stay as they are until the next step, in pinned memory too.

Two chunks are in flight at once: the later one's image must not reach the
buffer while the reader still looks at the earlier one's. The images are large
enough for pinned memory and the reader takes longer than a chunk.
"""
import time

import numpy as np
import pytest

from meercadraytracer_b200 import pinned

pytestmark = pytest.mark.gpu

W, H, SAMPLES = 256, 192, 12


@pytest.fixture(scope="module")
def small():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    return compile_with_oracle(b.scene), compile_camera(b.camera), trace_settings({"global_illumination": True})


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("passes", [1, 2])
def test_a_slow_reader_sees_the_image_its_event_names(small, passes, use_graph):
    from meercadraytracer_b200.batch import EVENT_DONE, EVENT_PREVIEW, EVENT_PROGRESS, BatchRenderer, RenderRequest
    from meercadraytracer_b200.executors import GpuExecutor

    compiled, cam, st = small
    ex = GpuExecutor(0)
    renderer = BatchRenderer(0, capacity=2 * passes * W * H, memory_budget=64 << 20, use_graph=use_graph)
    try:
        want = {n: ex.raytrace(compiled, cam, W, H, st, n, True).copy() for n in range(passes, SAMPLES + 1, passes)}
        # Dropped results earn pinned blocks: until the request's three images get them.
        for _ in range(20):
            blocks = [pinned.empty(W * H * 4, np.uint8) for _ in range(3 + 2 * pinned.FRESH)]
            del blocks
        rid = renderer.submit(RenderRequest(compiled, cam, W, H, st, SAMPLES, 4, progress=True))
        assert renderer.progress(rid).base is not None  # pinned
        seen, previews = [], 0
        for _ in range(100):
            events, idle = renderer.step()
            shown = {EVENT_PREVIEW: renderer.preview, EVENT_PROGRESS: renderer.progress, EVENT_DONE: renderer.result}
            at_once = [shown[kind](rid).copy() for _, kind, _ in events]
            time.sleep(0.02)
            for (_, kind, n), image in zip(events, at_once):
                assert np.array_equal(shown[kind](rid), image)
                previews += kind == EVENT_PREVIEW
                if kind != EVENT_PREVIEW:
                    assert np.array_equal(image, want[n])
                    seen.append(n)
            if idle:
                break
        assert seen == sorted(want) and previews == 1
    finally:
        renderer.dispose()
        ex.dispose()
