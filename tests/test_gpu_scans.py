"""The scans and lists between the stages where their kernels change: scans of
one block, of tiles whose blocks add up the tiles before them, and with a kernel
that scans the tiles' sums first; band lists by a warp per word and by a lane per
word.  All whole numbers, compared exactly (with numpy, or with the FP32 oracle
through the parity tests)."""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_parity import _run

pytestmark = pytest.mark.gpu

TILE, SUMS = 4096, 16384


@pytest.mark.parametrize("n", [1, TILE - 1, TILE, TILE + 1, 4 * TILE, 4 * TILE + 1, 300 * TILE + 5, SUMS * TILE,
                               SUMS * TILE + 1])
def test_exclusive_scan(n):
    import torch
    from fluidsurfacereconstructiongpu_gb300 import _native as N
    scan = N.lib.launchThrustExclusivePrefixSumScan
    scan.restype = ctypes.c_uint32
    scan.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32]
    x = np.random.default_rng(n % 1000).integers(0, 1 << 32, n, dtype=np.uint32)
    d = torch.from_numpy(x.view(np.int32)).cuda()
    out = torch.zeros_like(d)
    want = np.cumsum(x, dtype=np.uint32)  # modulo 2^32, as the device's
    torch.cuda.synchronize()
    total = scan(out.data_ptr(), d.data_ptr(), n)
    got = out.cpu().numpy().view(np.uint32)
    assert total == want[-1] and got[0] == 0 and np.array_equal(got[1:], want[:-1])
    assert scan(d.data_ptr(), d.data_ptr(), n) == total  # in place
    assert torch.equal(d, out)


def _slabs(h, n, seed):
    """Particles in two thin slabs and a few on their own: empty words, words of
    one vertex, rows that start and end inside a word."""
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    rng = np.random.default_rng(seed)
    pos = rng.random((n, 3))
    pos[: n // 2, 0] = 0.2 + 0.05 * pos[: n // 2, 0]
    pos[n // 2: n - 20, 1] = 0.6 + 0.05 * pos[n // 2: n - 20, 1]
    return synthetic.ParticleFrame(bbox_min=np.zeros(3, np.float32), bbox_max=np.ones(3, np.float32), h=h,
                                   particle_radius=h / 4, mass=1000.0 * (h / 4) ** 3, pos=pos.astype(np.float32),
                                   density=np.full(n, 1000.0, np.float32))


# grids of 41^3, 61^3, 81^3 (one block / tiles: 16,384 words = 80.6^3), 161^3 and 162^3 vertices (130,415 and
# 132,861 words, on both sides of the lists' line), and 241^3
@pytest.mark.parametrize("cells,ratio", [(20, 2), (20, 3), (20, 4), (20, 8), (23, 7), (24, 10)])
@pytest.mark.parametrize("method", ["tc01", "yu13"])
def test_band_lists_and_offsets(method, cells, ratio):
    h = 1.0 / (cells - 0.4)  # a cell per h
    _run(method, _slabs(h, 3000, cells + ratio), grid_ratio=ratio, cell_size_scale=1.0,
         iso=0.1 if method == "tc01" else -0.4)
