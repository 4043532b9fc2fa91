"""dL/dx of the grouped ZB05 / TC01 adjoint against PyTorch autograd in 64 bits
on the same topology, where the kernel's bookkeeping changes: groups of few and
of more than 128 vertices with a gradient (fine grids), windows of a few
particles and of several staged segments, frames of few groups (z slabs) and of
many.  The mesh's edges come from the weld keys (3 x lower grid vertex + axis);
the bar is the finite-difference tests' (2e-3 of the largest gradient)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(n, h, spread, seed):
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    rng = np.random.default_rng(seed)
    pos = (0.5 + spread * (rng.random((n, 3)) - 0.5)).astype(np.float32)
    return synthetic.ParticleFrame(bbox_min=np.zeros(3, np.float32), bbox_max=np.ones(3, np.float32), h=h,
                                   particle_radius=h / 4, mass=1.0, pos=pos, density=np.full(n, 1000.0, np.float32))


def _vertices(rec, fr, ratio):
    """Grid end points (positions in 64 bits) of each soup vertex's edge."""
    import torch
    s = rec.stats()
    key = torch.from_numpy(rec.debug("weld_keys").astype(np.int64)).cuda()
    low, axis = key // 3, key % 3
    rx, ry = int(s.scalar_res[0]), int(s.scalar_res[1])
    idx = torch.stack([low % rx, low // rx % ry, low // (rx * ry)], 1)
    other = idx.clone()
    other[torch.arange(len(key), device="cuda"), axis] += 1
    cs = np.float32(fr.h)  # cell = h
    scs = float(cs / np.float32(ratio))
    lo = torch.tensor([float(np.float32(b) - cs) for b in fr.bbox_min], device="cuda", dtype=torch.float64)
    return idx * scs + lo, other * scs + lo


@pytest.mark.parametrize("method", ["zb05", "tc01"])
@pytest.mark.parametrize("n,h,spread,ratio", [(1, 0.1, 0.1, 8), (40, 0.1, 0.25, 2), (40, 0.1, 0.9, 8),
                                              (500, 0.1, 0.25, 12), (900, 0.12, 0.2, 5), (2500, 0.05, 0.4, 8)])
def test_gradient_matches_autograd(method, n, h, spread, ratio):
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api
    fr = _frame(n, h, spread, n)
    xyz, den, iso = torch.from_numpy(fr.pos).cuda(), torch.from_numpy(fr.density).cuda(), -0.0001
    if method == "tc01":  # a level that the band has on both sides: the median of its field
        rec = api.Reconstructor(method, 0, grid_ratio=ratio)
        rec.reconstruct(xyz, den, api.header_of(fr))
        iso = float(np.median(rec.debug("field")))
        rec.close()
    rec = api.Reconstructor(method, 0, weld=True, grid_ratio=ratio, iso=iso)
    nv = rec.reconstruct(xyz, den, api.header_of(fr))
    assert nv > 0
    pos, _ = rec.mesh_tensors()
    g = torch.randn(nv, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    got = rec.backward(g).double()
    x = torch.from_numpy(fr.pos).cuda().double().requires_grad_(True)
    pa, pb = _vertices(rec, fr, ratio)
    rec.close()
    h2, rp = float(np.float32(fr.h)) ** 2, float(np.float32(fr.particle_radius))

    def field(v):
        out = []
        for part in v.split(20000):
            d = x[None] - part[:, None]
            t = d.square().sum(2) / h2
            if method == "tc01":
                out.append(torch.where(t <= 1, (t / 2) ** 2 - t / 2 + 0.25, 0.0).sum(1))
            else:
                w = (1 - t).clamp(min=0) ** 3
                ws = w.sum(1)
                m = (w[:, :, None] * d).sum(1) / torch.where(ws > 0, ws, 1.0)[:, None]
                out.append(torch.where(ws > 0, m.square().sum(1).clamp(min=1e-30).sqrt() - rp, 0.0))
        return torch.cat(out)

    # each edge once: a soup holds an edge several times
    both, where = torch.unique(torch.cat([pa, pb]), dim=0, return_inverse=True)
    phi = field(both)
    fa, fb = phi[where[:nv]], phi[where[nv:]]
    d = fb - fa
    keep = d.detach().abs() > 1e-7
    f = torch.where(keep, (float(np.float32(iso)) - fa) / torch.where(keep, d, 1.0), 0.5)
    p = pa + f[:, None] * (pb - pa)
    assert (p.detach() - pos.double()).abs().max() < 1e-4 * h
    want, = torch.autograd.grad((p * g.double()).sum(), x)
    assert (got - want).abs().max() <= 2e-3 * want.abs().max()


@pytest.mark.parametrize("ratio", [4, 5])
def test_anisotropic_adjoint_by_runs_and_by_slabs(ratio):
    """The anisotropic field's adjoint on both sides of the line between work
    items by runs of candidates (up to 4 vertices per cell) and by slabs of
    vertices, at the bar of the finite-difference tests."""
    from fluidsurfacereconstructiongpu_gb300 import synthetic
    from tests.test_gpu_backward import ANISO_SETTINGS, _case
    fr = synthetic.lattice_cube(12, 0.0125, seed=1, origin=(0.3, 0.3, 0.3))
    rows, err, scale = _case("yu13", fr, **dict(ANISO_SETTINGS["fine"], grid_ratio=ratio))
    assert scale > 0
    assert err.max() <= 2e-3 * scale, (err.max() / scale, rows[np.argmax(err)])
