"""Host images of a batch's requests live for as long as the engine may write them.

CPU: the binding over a stand-in for the engine. GPU: a call that fails leaves
nothing of its requests behind, queued or in flight.
"""
import gc
import weakref

import numpy as np
import pytest

from meercadraytracer_b200 import batch as B
from meercadraytracer_b200._lib import McrtError


class Engine:
    """What BatchRenderer calls, with requests that end when the test says so."""

    def __init__(self):
        self.held = set()
        self.next_id = 1
        self.fail_render = False

    def call(self, name, *args):
        if name == "mcrt_batch_create":
            args[-1]._obj.value = 1
        elif name == "mcrt_batch_submit":
            args[2]._obj.value = self.next_id
            self.held.add(self.next_id)
            self.next_id += 1
        elif name == "mcrt_batch_holds":
            args[2]._obj.value = int(args[1] in self.held)
        elif name == "mcrt_batch_render" and self.fail_render:
            raise RuntimeError("a request was refused")


class Scene:
    class _h:
        value = 1


@pytest.fixture
def engine(monkeypatch):
    e = Engine()
    monkeypatch.setattr(B, "call", e.call)
    monkeypatch.setattr(B, "load", lambda: None)
    monkeypatch.setattr(B.BatchRenderer, "_c_fields", staticmethod(lambda *a: B.abi.mcrt_request()))
    return e


def test_a_forgotten_requests_images_wait_for_the_engine(engine):
    r = B.BatchRenderer()
    rid = r.submit_to(Scene(), (1, 1), None, None, 32, 32, 4, progress=True)
    images = [weakref.ref(a) for a in (r.result(rid), r.progress(rid))]
    r.forget(rid)
    for _ in range(10):  # still queued: however many steps that takes
        r.step()
        gc.collect()
        assert all(w() is not None for w in images)
    engine.held.clear()
    r.step()
    gc.collect()
    assert all(w() is None for w in images)


def test_images_of_ended_requests_go_at_once(engine):
    r = B.BatchRenderer()
    rid = r.submit_to(Scene(), (1, 1), None, None, 32, 32, 4)
    image = weakref.ref(r.result(rid))
    engine.held.clear()
    r.forget(rid)
    gc.collect()
    assert image() is None


def test_render_releases_what_ended_meanwhile(engine):
    r = B.BatchRenderer()
    rid = r.submit_to(Scene(), (1, 1), None, None, 32, 32, 4)
    image = weakref.ref(r.result(rid))
    r.forget(rid)
    engine.held.clear()
    engine.fail_render = True
    with pytest.raises(RuntimeError):
        r.render([])
    gc.collect()
    assert image() is None and not r._retired


@pytest.fixture(scope="module")
def small():
    from helpers import compile_with_oracle
    from meercadraytracer_b200 import scenes
    from meercadraytracer_b200.compile import compile_camera
    from meercadraytracer_b200.raytrace import trace_settings

    b = scenes.small_scene()
    return compile_with_oracle(b.scene), compile_camera(b.camera), trace_settings({})


@pytest.mark.gpu
def test_a_refused_batch_leaves_no_request_behind(small):
    compiled, cam, st = small
    good, bad = B.RenderRequest(compiled, cam, 64, 48, st, 3), B.RenderRequest(compiled, cam, 64, 48, st, 0)
    r = B.BatchRenderer(0, capacity=1 << 14, memory_budget=16 << 20)
    try:
        (want,) = r.render([good])
        traced = r.stats()["samples"]
        with pytest.raises(McrtError):
            r.render([good, good, bad])
        assert r.step() == ([], True)
        assert r.stats()["samples"] == traced and r.stats()["arena_used"] == 0
        (again,) = r.render([good])
        assert np.array_equal(again, want)
    finally:
        r.dispose()


@pytest.mark.gpu
def test_a_batch_that_fails_on_the_way_leaves_nothing_in_flight(small):
    compiled, cam, st = small
    r = B.BatchRenderer(0, capacity=1 << 14, memory_budget=16 << 20, use_graph=False)
    try:
        good = B.RenderRequest(compiled, cam, 64, 48, st, 12)
        (want,) = r.render([good])
        ex = r.executor(compiled)
        ex.set_step_limit(3)
        fresh = B.BatchRenderer(0, capacity=1 << 14, memory_budget=16 << 20, use_graph=False)
        try:
            fresh.adopt(compiled, ex)
            with pytest.raises(McrtError):
                fresh.render([good])
            assert fresh.step() == ([], True) and fresh.stats()["arena_used"] == 0
        finally:
            fresh.dispose()
            ex.set_step_limit(0)
        (again,) = r.render([good])
        assert np.array_equal(again, want)
    finally:
        r.dispose()
