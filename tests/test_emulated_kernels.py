"""Kernels run on the host lane by lane (tests/cpp/warp_emul.h)."""
import pytest

from tests import emulated


def test_tile_order_does_not_depend_on_the_order_of_atomics():
    """The two warps of a split work item lay out the same pass each for itself
    and write every second tile: a vertex must have one place."""
    assert emulated.run("tile_order") == "same\n"


@pytest.mark.parametrize("what", ["stamp", "group", "blocks", "classify"])
def test_counts_above_two_to_the_31(what):
    """Sizes that frame_plan accepts: no index wraps, every loop ends."""
    got = emulated.run("big_counts", what, timeout=60)
    if got == "no address space\n":
        pytest.skip("cannot reserve the arrays' address space")
    assert got == "ok\n"


def test_smoothing_by_four_lanes_joins_its_chunk_sums_like_the_one_lane_kernel():
    """Also chunks of 32 candidates that all lie beyond the radius, whose sum of
    0 a compensated total still takes."""
    assert emulated.run("smooth_sums") == "differing means 0, FP32 means 0, smoothed positions 0\n"


def test_adjoints_of_vertices_that_are_not_finite():
    """A NaN or infinite dL/dphi reaches the particles in whose support the
    vertex lies, as a range test has it, and no others."""
    assert emulated.run("adjoints", "nan") == "ok\n"


def test_anisotropic_adjoint_where_the_first_sums_cancel():
    """dL/dG of a particle whose sums of b d and g u^3 vanish exactly."""
    assert emulated.run("adjoints", "cancel") == "ok\n"


def test_adjoints_of_groups_that_warps_share():
    """Runs of candidates, usual and crowded groups."""
    assert emulated.run("adjoints", "shared") == "ok\n"
