"""The ZB05 adjoint where a window holds many particles: groups whose
candidates several warps share (coarse grids, crowded cells), against autograd in
64 bits at the grouped adjoint's bar, and its time against the frame's."""
import pytest

from tests import test_gpu_backward_groups as groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ratio", [(600, 2), (6000, 2), (6000, 4), (6000, 8)])
def test_gradient_matches_autograd(n, ratio):
    """Eight cells of 75 or of 750 particles (crowded: 256 a cell and more).  (TC01
    shares the code; tests/cpp/adjoints.cpp compares both per pair.)"""
    groups.test_gradient_matches_autograd("zb05", n, 0.1, 0.2, ratio)


def test_backward_of_dense_cells_takes_a_fraction_of_the_frame():
    """30,000 particles, 1000 a cell, on the default grid: with a warp per group
    0.6 of the frame's time, with the groups shared 0.1."""
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api
    fr = groups._frame(30000, 0.32, 1.0, 3)
    xyz, den = torch.from_numpy(fr.pos).cuda(), torch.from_numpy(fr.density).cuda()
    rec = api.Reconstructor("zb05", 0)
    header = api.header_of(fr)

    def best(call):
        times = []
        for _ in range(8):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            call()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times[3:])

    frame = best(lambda: rec.reconstruct(xyz, den, header))
    g = torch.ones((rec.reconstruct(xyz, den, header), 3), device="cuda")
    assert len(g) > 0
    back = best(lambda: rec.backward(g))
    rec.close()
    assert back < 0.3 * frame, (back, frame)
