"""The capacity rule after an unchecked frame: room for a growing scene, never
more than a call takes."""
import pytest

from ubs.render import MAX_CAPACITY, Renderer


class _Stats:
    def __init__(self, total):
        self.total = total

    def wait(self):
        return self.total, 0


@pytest.mark.parametrize("total, cap, want", [
    (100, 1000, 1000),                                # plenty of room
    (900, 1000, int(900 * 1.25) + 1024),              # within an eighth of the capacity
    (1_720_000_000, 1_800_000_000, MAX_CAPACITY),     # 25% more is past the limit
    (MAX_CAPACITY - 5, MAX_CAPACITY, MAX_CAPACITY),
])
def test_capacity_after_a_frame_that_fits(total, cap, want):
    r = Renderer(dim=6, capacity=cap)
    r._pending = (_Stats(total), cap)
    r._check_pending()
    assert r.capacity == want <= 2 ** 31 - 1
    assert r.last_isects == total


def test_overflow_is_still_reported():
    r = Renderer(dim=6, capacity=1000)
    r._pending = (_Stats(1001), 1000)
    with pytest.raises(RuntimeError, match="capacity is now"):
        r._check_pending()
    assert r.capacity == int(1001 * 1.25) + 1024
