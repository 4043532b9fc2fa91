"""Kernels run on the host lane by lane (tests/cpp/warp_emul.h)."""
from tests import emulated


def test_tile_order_does_not_depend_on_the_order_of_atomics():
    """The two warps of a split work item lay out the same pass each for itself
    and write every second tile: a vertex must have one place."""
    assert emulated.run("tile_order") == "same\n"
