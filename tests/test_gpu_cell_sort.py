"""Spatial hashing by counting sort: sort order, cell ranges and sorted
positions must equal a stable sort of the FP32 cell keys, for one particle up to
many, cells of one particle up to crowds (on both sides of 1,024 particles a
cell, which a block sorts), arrival orders of every kind, and on both sides of
the rule that leaves sparse grids to the radix sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(pos, h):
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api
    pos = np.ascontiguousarray(pos, np.float32)
    n = len(pos)
    lo, hi = np.zeros(3, np.float32), np.ones(3, np.float32)
    rec = api.Reconstructor("zb05", 0, grid_ratio=1)
    rec.reconstruct(torch.from_numpy(pos).cuda(), torch.ones(n, device="cuda"),
                    api.header_from(lo, hi, h, h / 4, 1.0))
    perm, srt, ranges = rec.debug("perm"), rec.debug("sorted_xyz"), rec.debug("ranges")
    res = [int(v) for v in rec.stats().spatial_res]
    rec.close()
    cs = np.float32(h)
    mn = lo - cs
    c = ((pos - mn) / cs).astype(np.int64)  # FP32 difference and quotient, truncated
    key = (c[:, 2] * res[1] + c[:, 1]) * res[0] + c[:, 0]
    want = np.argsort(key, kind="stable")
    assert np.array_equal(perm, want)
    assert np.array_equal(srt, pos[want])
    cells = res[0] * res[1] * res[2]
    count = np.bincount(key, minlength=cells)
    end = np.cumsum(count)
    some = count > 0
    assert np.array_equal(ranges[some, 0], (end - count)[some])
    assert np.array_equal(ranges[some, 1], end[some])
    assert np.all(ranges[~some] == 0xFFFFFFFF)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 4097, 70001])
@pytest.mark.parametrize("h", [0.5, 0.06])
def test_uniform(n, h):
    _check(np.random.default_rng(n).random((n, 3)), h)


@pytest.mark.parametrize("crowd", [1023, 1024, 1025, 5000, 70000])
@pytest.mark.parametrize("order", ["random", "sorted", "blocks"])
def test_crowded_cells(crowd, order):
    rng = np.random.default_rng(crowd)
    a = 0.3 + 0.01 * rng.random((crowd, 3))
    b = 0.7 + 0.01 * rng.random((crowd + 3, 3))
    pos = np.concatenate([a, b, rng.random((3000, 3))])
    if order == "random":
        pos = pos[rng.permutation(len(pos))]
    elif order == "blocks":
        pos = np.concatenate([pos[k::7] for k in range(7)])
    _check(pos, 0.11)


@pytest.mark.parametrize("n", [1, 400, 13000, 14000])
def test_sparse_grid(n):
    """52^3 = 140,608 cells: 8 n + 16,384 reaches them at 15,528 particles."""
    _check(np.random.default_rng(n).random((n, 3)), 0.02)


@pytest.mark.parametrize("n", [15527, 15528])
def test_both_sides_of_the_rule(n):
    _check(np.random.default_rng(n).random((n, 3)), 0.02)
