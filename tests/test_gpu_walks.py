"""The neighbour walks of the anisotropic path, against the oracles, where
their choices change: a warp's lanes in one set of windows, in several (rows of
cells that end inside the warp) and scattered over the grid; neighbour radii
below and above a cell; the sizes on both sides of the lines between the kernels
(four lanes per particle or one); the smallest frames.  The bars are those of
the parity tests (FP32 means and counts exact, G and the field against FP64)."""
import numpy as np
import pytest

from tests.test_gpu_parity import _run

pytestmark = pytest.mark.gpu

# neighbour radius / cell: 0.8 (the benchmark's), 1.54 (the defaults'), 0.38 and 1.05 (multiples of h that
# the library and the oracle round alike)
SETTINGS = {
    "fine": dict(smoothing_lambda=0.9, aniso_radius_over_h=1.0, cell_size_scale=1.25, grid_ratio=4, iso=0.0),
    "default": {},
    "short": dict(smoothing_lambda=0.9, aniso_radius_over_h=0.5, cell_size_scale=1.3, grid_ratio=3),
    "over": dict(smoothing_lambda=0.5, aniso_radius_over_h=1.365, cell_size_scale=1.3, grid_ratio=3),
}


def _frame(n, h, spread, seed):
    """n particles uniform in a box of the given fraction of the unit cube."""
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    rng = np.random.default_rng(seed)
    pos = (0.5 + spread * (rng.random((n, 3)) - 0.5)).astype(np.float32)
    return synthetic.ParticleFrame(bbox_min=np.zeros(3, np.float32), bbox_max=np.ones(3, np.float32), h=h,
                                   particle_radius=h / 4, mass=1000.0 * (h / 4) ** 3, pos=pos,
                                   density=np.full(n, 1000.0, np.float32))


@pytest.mark.parametrize("settings", sorted(SETTINGS))
@pytest.mark.parametrize("n", [1, 7, 33, 1000])
def test_few_particles(n, settings):
    _run("yu13", _frame(n, 0.08, 0.3, n), **SETTINGS[settings])


@pytest.mark.parametrize("settings", ["fine", "default", "over"])
def test_scattered_particles(settings):
    """About one particle to two cells: every lane a window of its own."""
    _run("yu13", _frame(3000, 0.05, 0.95, 5), **SETTINGS[settings])


@pytest.mark.parametrize("settings", ["fine", "default", "over"])
def test_rows_of_few_cells(settings):
    """A slab two cells wide: most warps run over the ends of several rows."""
    fr = _frame(4000, 0.04, 0.9, 6)
    fr.pos[:, 0] = 0.5 + (fr.pos[:, 0] - 0.5) * 0.1
    _run("yu13", fr, **SETTINGS[settings])


@pytest.mark.parametrize("n_side,settings", [(36, "fine"), (37, "fine"), (43, "default"), (44, "default"),
                                             (23, "default"), (24, "default"), (50, "over"), (51, "over")])
def test_both_sides_of_the_lanes_per_particle_rule(n_side, settings):
    """46,656 / 50,653, 79,507 / 85,184, 12,167 / 13,824 and 125,000 / 132,651 particles."""
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    fr = synthetic.lattice_cube(n_side, 0.008, seed=n_side, jitter_frac=0.3, origin=(0.2, 0.2, 0.2))
    _run("yu13", fr, **SETTINGS[settings])


@pytest.mark.parametrize("case", ["lattice", "scattered", "slab"])
def test_smoothing_of_the_same_particles_by_both_kernels(case):
    """Below a cell's radius, four lanes per particle and one sum in the same
    order and the same chunks: particles that sort first smooth to the same bits
    whether 40,000 others further up bring the frame past the line or not."""
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api, synthetic
    fr = _frame(8000, 0.02, 0.5, 8)
    if case == "lattice":
        fr.pos = (0.3 + 0.2 * synthetic.lattice_cube(20, 0.025, seed=2, jitter_frac=0.3).pos).astype(np.float32)
    elif case == "slab":
        fr.pos[:, 0] = 0.5 + (fr.pos[:, 0] - 0.5) * 0.1
    fr.pos[:, 2] = 0.1 + 0.5 * (fr.pos[:, 2] - fr.pos[:, 2].min())
    n = len(fr.pos)
    far = np.random.default_rng(9).random((49152 - n + 100, 3)) * [0.9, 0.9, 0.2] + [0.05, 0.05, 0.75]
    got = []
    for pos in (fr.pos, np.concatenate([fr.pos, far.astype(np.float32)])):
        rec = api.Reconstructor("yu13", 0, keep_intermediates=True, **SETTINGS["fine"])
        fr.density = np.full(len(pos), 1000.0, np.float32)
        rec.reconstruct(torch.from_numpy(pos).cuda(), torch.from_numpy(fr.density).cuda(), api.header_of(fr))
        got.append((np.array(rec.debug("perm"))[:n], np.array(rec.debug("smoothed"))[:n]))
        rec.close()
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("scale", [1.0, 1.4])
@pytest.mark.parametrize("case", ["few1", "few40", "scattered", "slab", "duplicates", "below", "above"])
def test_colour_field_walks(case, scale):
    """The Akinci12 colour field by four lanes per particle and by one (97,336 /
    103,823 particles); windows in one set, in several, scattered; particles on
    top of one another (at distance 0, not counted).  The flags are exact (the
    field is not looked at: isolated vertices' weights are ill-conditioned)."""
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    if case.startswith("few"):
        fr = _frame(int(case[3:]), 0.08, 0.3, 3)
    elif case == "scattered":
        fr = _frame(3000, 0.05, 0.95, 5)
    elif case == "slab":
        fr = _frame(4000, 0.04, 0.9, 6)
        fr.pos[:, 0] = 0.5 + (fr.pos[:, 0] - 0.5) * 0.1
    elif case == "duplicates":
        fr = _frame(1500, 0.06, 0.3, 7)
        fr.pos[1::3] = fr.pos[::3]
    else:
        fr = synthetic.lattice_cube(46 if case == "below" else 47, 0.008, seed=9, jitter_frac=0.3,
                                    origin=(0.2, 0.2, 0.2))
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api
    from oracle import pipeline as P
    rec = api.Reconstructor("akinci", 0, keep_intermediates=True, cell_size_scale=scale, grid_ratio=2)
    rec.reconstruct(torch.from_numpy(fr.pos).cuda(), torch.from_numpy(fr.density).cuda(), api.header_of(fr))
    params = P.FrameParams(method="akinci", h=fr.h, particle_radius=fr.particle_radius, mass=fr.mass,
                           cell_scale=scale, ratio=2)
    o32 = P.run_frame("oracle32", fr.pos, fr.density, fr.bbox_min, fr.bbox_max, params)
    assert np.array_equal(rec.debug("surface_flags"), o32.sflag)
    assert np.array_equal(rec.debug("band"), o32.sv)
    rec.close()


@pytest.mark.parametrize("scale", [0.7, 1.0, 1.4])
@pytest.mark.parametrize("case", ["few1", "few40", "scattered", "slab", "dense"])
def test_density_walks(case, scale):
    """Windows of one, several and many sets of lanes, cells smaller than h."""
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api
    from oracle.pipeline import sph_density
    if case.startswith("few"):
        fr = _frame(int(case[3:]), 0.08, 0.3, 3)
    elif case == "dense":
        fr = _frame(3001, 0.08, 0.3, 4)
    else:
        fr = _frame(3000, 0.05, 0.95, 5)
        if case == "slab":
            fr.pos[:, 0] = 0.5 + (fr.pos[:, 0] - 0.5) * 0.1
    rec = api.Reconstructor("zb05", 0, compute_density=True, cell_size_scale=scale)
    rec.reconstruct(torch.from_numpy(fr.pos).cuda(), None, api.header_of(fr))
    got = rec.debug("density").astype(np.float64)
    perm = rec.debug("perm")
    rec.close()
    want = sph_density(fr.pos, fr.h, fr.mass)[perm]
    assert np.all(np.abs(got - want) <= 1e-5 * want)
