"""The autotuner times each traversal kernel once: pairs of one block size name the same one."""
from types import SimpleNamespace

import pytest

from meercadraytracer_b200 import autotune

PAIRS = [(128, 4), (128, 8), (64, 16), (128, 16), (256, 8), (256, 16)]
MS = {128: 2.0, 64: 3.0, 256: 1.0}


class Timed:
    """An executor and a batch whose times go by the block size alone, each run a little longer than the last."""

    device, capacity = 0, 1 << 20

    def __init__(self):
        self.block, self.ms, self.runs = 128, 0.0, []

    def set_traversal(self, block, stack):
        self.block = block

    def set_capacity(self, paths):
        pass

    set_chunk = set_capacity

    def reset_stats(self):
        self.ms = 0.0

    def raytrace(self, *args):
        self.runs.append(self.block)
        self.ms += MS[self.block] + 1e-3 * len(self.runs)

    def render(self, requests):
        self.raytrace()

    def stats(self):
        return {"ms_total": self.ms, "gpu_ms": self.ms}


@pytest.fixture(autouse=True)
def nothing_cached(monkeypatch):
    monkeypatch.setattr(autotune, "_memory", {})


@pytest.mark.parametrize("best,pairs", [((256, 8), PAIRS), ((128, 4), PAIRS[:4]), ((64, 16), [(64, 16)])])
def test_plain(best, pairs):
    ex = Timed()
    scene = SimpleNamespace(geometry=SimpleNamespace(triangle_count=1))
    c = autotune.tune_plain(ex, scene, None, None, 8, 8, 1, capacities=(1,), variants=pairs, repeats=1, key="k")
    blocks = [b for i, (b, _) in enumerate(pairs) if b not in [p[0] for p in pairs[:i]]]
    assert ex.runs[1:-1] == blocks  # after the warm-up, before the one capacity
    assert (c.block, c.stack) == best == (ex.block, c.stack)
    assert [t for t in c.timings if t.startswith("variant")] == [f"variant {b}x{s}" for b, s in pairs]


def test_batch():
    r = Timed()
    c = autotune.tune_batch(r, [None], chunks=(1,), variants=PAIRS, key="k")
    assert r.runs[1:-1] == [128, 64, 256] and (c.block, c.stack) == (256, 8)
