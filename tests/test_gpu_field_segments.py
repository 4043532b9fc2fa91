"""The grouped ZB05 / TC01 fields stage candidates in segments and go through
the tiles of a pass per segment: windows of few particles up to several
segments' worth, groups of one tile (coarse grids) and of several, frames with
groups cut into slabs, against the oracles (the parity tests' bars)."""
import numpy as np
import pytest

from tests.test_gpu_parity import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["zb05", "tc01", "akinci"])
@pytest.mark.parametrize("per_cell,ratio", [(0.2, 8), (4, 1), (4, 8), (4.6, 3), (13, 5), (40, 2), (40, 11)])
def test_window_sizes(method, per_cell, ratio):
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    h, side = 0.08, 4.3
    n = int(per_cell * side ** 3)
    rng = np.random.default_rng(int(10 * per_cell) + ratio)
    pos = (0.41 + h * side * (rng.random((n, 3)) - 0.5)).astype(np.float32)
    fr = synthetic.ParticleFrame(bbox_min=np.zeros(3, np.float32), bbox_max=np.ones(3, np.float32), h=h,
                                 particle_radius=h / 4, mass=1000.0 * h ** 3 / per_cell, pos=pos,
                                 density=np.full(n, 1000.0, np.float32))
    _run(method, fr, grid_ratio=ratio)
