"""New pinned blocks go to programs whose blocks come back, ordinary memory to those that keep their results."""
import gc

import numpy as np
import pytest

from meercadraytracer_b200 import pinned
from test_host_memory import HostPool


def pinned_count(arrays):
    return sum(a.base is not None for a in arrays)


@pytest.mark.parametrize("rounds", [1, 5, 40])
def test_kept_results_stop_taking_new_blocks(monkeypatch, rounds):
    pool = HostPool(monkeypatch)
    kept = [pool.empty(1 << 20, np.uint8) for _ in range(rounds)]
    assert pinned_count(kept) == len(pool.blocks) == min(rounds, pinned.FRESH)


@pytest.mark.parametrize("images", [1, 2, 3, 12, 64])
def test_dropped_results_get_blocks_for_all(monkeypatch, images):
    pool = HostPool(monkeypatch)
    calls = 0
    while True:
        batch = [pool.empty(1 << 20, np.uint8) for _ in range(images)]
        have = pinned_count(batch)
        del batch
        gc.collect()
        if have == images:
            break
        calls += 1
        assert calls <= 7  # what returned lets at least as many again be new
    assert len(pool.blocks) == images


def test_keeping_after_dropping_is_bounded(monkeypatch):
    pool = HostPool(monkeypatch)
    for _ in range(100):
        pool.empty(1 << 20, np.uint8)
        gc.collect()
    kept = [pool.empty(1 << 20, np.uint8) for _ in range(50)]
    assert pinned_count(kept) == len(pool.blocks) <= 2 + pinned.FRESH


@pytest.mark.parametrize("images", [1, 3, 12])
def test_first_results_kept_and_later_ones_dropped(monkeypatch, images):
    pool = HostPool(monkeypatch)
    first = [pool.empty(1 << 20, np.uint8) for _ in range(images)]
    for calls in range(8):
        batch = [pool.empty(1 << 20, np.uint8) for _ in range(images)]
        have = pinned_count(batch)
        del batch
        gc.collect()
    assert have == images and pinned_count(first) == min(images, pinned.FRESH)
    assert len(pool.blocks) == images + pinned_count(first)
