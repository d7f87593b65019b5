"""Room made ahead for pinned blocks: what is allocated in it stands in it, and it goes back with its last block."""
import pytest

from meercadraytracer_b200._lib import call
from test_host_blocks import MB, alloc, free, gpu  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def mapping_of(a):
    """The process's mapping that holds a block's first byte, or None."""
    at = a.ctypes.data
    with open("/proc/self/maps") as f:
        for line in f:
            lo, hi = (int(x, 16) for x in line.split()[0].split("-"))
            if lo <= at < hi:
                return lo, hi
    return None


def test_blocks_are_cut_from_the_reservation(gpu):  # noqa: F811
    call("mcrt_host_reserve", 0, 32 * MB)
    call("mcrt_host_reserve", 0, 16 * MB)  # within the first
    first = alloc(20 * MB)
    free(first)
    held = [alloc(s) for s in (4 * MB, 65536, 8 * MB, 3 * MB)]
    lo, hi = min(a.ctypes.data for a in held), max(a.ctypes.data + a.size for a in held)
    assert hi - lo <= 32 * MB
    for i, a in enumerate(held):
        a[:] = i + 1
    call("mcrt_host_unreserve")
    assert all((a == i + 1).all() for i, a in enumerate(held))
    call("mcrt_host_unreserve")
    assert all((a == i + 1).all() for i, a in enumerate(held))  # blocks outlive the reservation
    for a in held:
        free(a)
    assert mapping_of(held[0]) is None


def test_a_larger_reservation_adds_to_a_smaller_one(gpu):  # noqa: F811
    call("mcrt_host_reserve", 0, 8 * MB)
    call("mcrt_host_reserve", 0, 24 * MB)
    held = [alloc(8 * MB), alloc(16 * MB)]
    held[0][:], held[1][:] = 1, 2
    assert (held[0] == 1).all()
    for _ in range(2):
        call("mcrt_host_unreserve")
    for a in held:
        free(a)
    assert mapping_of(held[0]) is None and mapping_of(held[1]) is None
