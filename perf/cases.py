"""The frames this framework reconstructs, as timed cases.

Each case is one call (or one short sequence of calls) that a program makes through the package's public front
end: a frame with device tensors in and out, a frame with host arrays in and out, a frame with its gradient, a
welded frame for an indexed mesh file, and a batch of frames.  Every output is what that program keeps: the
triangle soup (positions and normals), the indexed mesh, the gradients, in buffers of the program's own.

``exact`` gives the same outputs from plain torch in 64 bits.  What the method defines in 32 bits (the grids, cell
indices, grid vertex positions, the band's distance test) is taken in 32 bits; sums, matrices, fields, vertices,
normals and gradients are in 64.
"""
import math

import numpy as np
import torch

from fluidsurfacereconstructiongpu_gb300 import api, autograd, synthetic

# The settings the package's benchmark and batches use (grid spacing of half a particle radius), and the methods'
# own defaults (coarse grids; the anisotropic field with a neighbour radius of 2h).
SETTINGS = {
    ("zb05", "fine"): dict(grid_ratio=8),
    ("tc01", "fine"): dict(grid_ratio=8),
    ("akinci12", "fine"): dict(grid_ratio=8),
    ("yu13", "fine"): dict(smoothing_lambda=0.9, aniso_radius_over_h=1.0, cell_size_scale=1.25, grid_ratio=10, iso=0.0),
    ("zb05", "default"): {},
    ("tc01", "default"): {},
    ("akinci12", "default"): {},
    ("yu13", "default"): {},
}
# What the defaults are, for exact() and work(): iso, vertices per cell, cell / h, lambda, neighbour radius / h.
DEFAULTS = {
    "zb05": (-0.0001, 2, 1.0, 0.0, 0.0),
    "tc01": (0.25, 2, 1.0, 0.0, 0.0),
    "akinci12": (-0.0001, 2, 1.0, 0.0, 0.0),
    "yu13": (0.0, 3, 1.3, 0.5, 2.0),
}
MIN_NEIGHBORS = 25
BATCH_METHODS = ("zb05", "yu13", "akinci12", "tc01")


def listed():
    return [
        # a preview of a small drop on the coarse default grid: launches and latency
        dict(name="zb05_drop_1k", use="frame", method="zb05", settings="default", scene="sphere", n=1500),
        # the small benchmark frame: a 32^3 block on the fine grid
        dict(name="zb05_block_32k", use="frame", method="zb05", settings="fine", scene="block", n=32768),
        # a simulator's frame in host arrays, the mesh back in host arrays (odd count)
        dict(name="tc01_host_100k", use="host", method="tc01", settings="default", scene="dam", n=100003),
        # the colour-field surface detection at a usual size
        dict(name="akinci_dam_262k", use="frame", method="akinci12", settings="fine", scene="dam", n=1 << 18),
        # the plain path at a million particles
        dict(name="zb05_dam_1m", use="frame", method="zb05", settings="fine", scene="dam", n=1 << 20),
        # the anisotropic method with its own defaults: neighbour radius 2h, coarse grid, noisy particles
        dict(name="yu13_default_40k", use="frame", method="yu13", settings="default", scene="sphere", n=40001),
        # the headline frame: a dam break of a million particles, anisotropic field on the fine grid
        dict(name="yu13_dam_1m", use="frame", method="yu13", settings="fine", scene="dam", n=1 << 20),
        # the largest frame: eight million particles, a scalar grid of 1.06e9 vertices
        dict(name="yu13_block_8m", use="frame", method="yu13", settings="fine", scene="block", n=8000000),
        # fitting particles to a surface: forward, a loss on the mesh, the gradient of the positions
        dict(name="yu13_train_150k", use="train", method="yu13", settings="fine", scene="dam", n=150001),
        # the same for positions and particle radius through the plain field
        dict(name="zb05_train_500k", use="train", method="zb05", settings="fine", scene="dam", n=500000),
        # particles without a density column, an indexed mesh for a file
        dict(name="yu13_indexed_120k", use="indexed", method="yu13", settings="fine", scene="sphere", n=120011),
        # frames of several scenes and methods in one call
        dict(name="batch_12x10k_80k", use="batch", method="mixed", settings="fine", scene="block", n=80000, n_lo=10000,
             frames=12),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    use = rng.choice(["frame", "frame", "frame", "frame", "train", "train", "host", "indexed", "batch"])
    settings = rng.choice(["fine", "fine", "fine", "default"])
    if use == "batch":
        return dict(use=use, method="mixed", settings=settings, scene="block", n=size(20000, 150000),
                    n_lo=size(2000, 20000), frames=rng.randint(3, 16))
    method = rng.choice(["zb05", "yu13", "yu13", "akinci12", "tc01"])
    top = {"frame": 2000000, "train": 600000, "host": 300000, "indexed": 300000}[use]
    if settings == "default" and method == "yu13":  # two thousand neighbours per particle
        top = min(top, 100000)
    return dict(use=use, method=method, settings=settings, scene=rng.choice(["dam", "dam", "block", "sphere"]),
                n=size(1200, top))


# ------------------------------------------------------------------ the cases
def _scene(scene, n, seed):
    if scene == "dam":  # the radius follows the count: the same neighbourhoods at every size
        return synthetic.dam_break(n, r=0.004 * ((1 << 20) / n) ** (1.0 / 3.0), seed=seed)
    if scene == "sphere":
        return synthetic.sphere_ball(n, seed=seed, displace_frac=0.25)
    return synthetic.lattice_count(n, seed=seed)


def _batch_cases(case):
    """The batch's frames as cases: the sizes belong to the case, the particles to the seed."""
    out = []
    for i in range(case["frames"]):
        t = i / max(1, case["frames"] - 1)
        n = int(round(math.exp(math.log(case["n_lo"]) * (1 - t) + math.log(max(case["n"], case["n_lo"])) * t)))
        out.append(dict(use="frame", method=BATCH_METHODS[i % 4], settings=case["settings"], scene=case["scene"], n=n))
    return out


def _batch_frames(case, seed):
    rng = np.random.default_rng(seed)
    return [(c["method"], _scene(c["scene"], c["n"], int(rng.integers(1 << 30)))) for c in _batch_cases(case)]


def prepare(case, seed):
    """The program's handle, particles and output buffers (of a size that the case alone sets, like a renderer's
    vertex buffer; the rows past the mesh stay zero)."""
    use, method = case["use"], case["method"]
    if use == "batch":
        frames = [(m, torch.from_numpy(f.pos).cuda(), torch.from_numpy(f.density).cuda(), api.header_of(f))
                  for m, f in _batch_frames(case, seed)]
        over = {m: SETTINGS[m, case["settings"]] for m in BATCH_METHODS}
        rooms = [_room(dict(c, use="frame")) for c in _batch_cases(case)]
        return dict(use=use, batch=api.Batch(0, params=over), frames=frames,
                    out=[[np.zeros((room, 3), np.float32) for _ in range(2)] for room in rooms])
    f = _scene(case["scene"], case["n"], seed)
    rec = api.Reconstructor(method, 0, weld=use == "indexed", compute_density=use == "indexed",
                            **SETTINGS[method, case["settings"]])
    room = _room(case)
    s = dict(use=use, rec=rec, header=api.header_of(f), room=room)
    if use in ("host", "indexed"):
        s["out"] = [np.zeros((room, 3), np.float32) for _ in range(2)]
    else:
        s["out"] = [torch.zeros((room, 3), device="cuda") for _ in range(1 if use == "train" else 2)]
    if use == "indexed":
        s["out"].append(np.zeros((room, 3), np.int32))
    if use == "host":
        return dict(s, xyz=f.pos, density=f.density)
    s["xyz"] = torch.from_numpy(f.pos).cuda()
    s["density"] = torch.from_numpy(f.density).cuda()
    if use == "train":
        s["xyz"].requires_grad_(True)
        s["radius"] = torch.tensor(f.particle_radius, device="cuda", requires_grad=True) if method == "zb05" else None
    return s


def run(s):
    use, out = s["use"], s["out"]
    if use == "batch":
        b = s["batch"]
        b.reconstruct(s["frames"])
        got = []
        for i in range(b.count):
            m = b.mesh(i)
            got.append([_put(m.positions, out[i][0]), _put(m.normals, out[i][1]), m.positions.shape[0]])
        return got
    rec = s["rec"]
    if use == "host":
        m = rec.reconstruct_host(s["xyz"], s["density"], s["header"], capacity=s["room"])
        return [_put(m.positions, out[0]), _put(m.normals, out[1]), m.positions.shape[0]]
    if use == "indexed":
        rec.reconstruct(s["xyz"], None, s["header"])
        m = rec.indexed_mesh()
        return [_put(m.positions, out[0]), _put(m.normals, out[1]), _put(m.triangles.view(np.int32), out[2]),
                m.positions.shape[0], m.triangles.shape[0]]
    if use == "train":
        xyz, radius = s["xyz"], s["radius"]
        pos = autograd.reconstruct_surface(xyz, s["density"], rec, s["header"], radius)
        _loss(pos).backward()
        got = [_put(pos.detach(), out[0]), xyz.grad, pos.shape[0]]
        xyz.grad = None
        if radius is not None:
            got.append(radius.grad)
            radius.grad = None
        return got
    n = rec.reconstruct(s["xyz"], s["density"], s["header"])
    pos, nrm = rec.mesh_tensors()
    return [_put(pos, out[0]), _put(nrm, out[1]), n]


def _put(rows, buffer):
    buffer[:rows.shape[0]] = rows
    return buffer


def _loss(pos):
    """The mesh against a sphere about the box's centre."""
    return ((pos - 0.5).square().sum(1) - 0.09).square().mean()


def _geometry(case):
    """Spacing, kernel radius, particle radius, scalar grid spacing, area of the scene's bodies, isolated particles."""
    n = case["n"]
    lone = 0.0
    if case["scene"] == "dam":  # column and droplet on a lattice, the rest is splash
        r = 0.004 * ((1 << 20) / n) ** (1.0 / 3.0)
        s = ((0.128 + 4.0 / 3.0 * math.pi * 0.08 ** 3) / (0.98 * n)) ** (1.0 / 3.0)
        area = 1.7
        lone = max(0.01 * n, n - round(0.4 / s) ** 2 * round(0.8 / s) - 4.0 / 3.0 * math.pi * (0.08 / s) ** 3)
    elif case["scene"] == "sphere":
        r = s = (4.0 / 3.0 * math.pi * 0.3 ** 3 / n) ** (1.0 / 3.0)
        area = 1.4
    else:
        r = s = 0.4 / n ** (1.0 / 3.0)
        area = 1.1
    _, ratio, scale, _, _ = _params(case["method"], case["settings"])
    return s, 4 * r, r, scale * 4 * r / ratio, area, lone


def _mesh_size(case):
    """Mesh vertices, about: two triangles for each grid square of the surface."""
    s, h, r, g, area, lone = _geometry(case)
    reach = 0.6 * h if case["use"] == "indexed" else r if case["method"] in ("zb05", "akinci12") else 0.0
    # the coarse TC01 surface follows single particles
    rough = 4.0 if case["method"] == "tc01" and case["settings"] == "default" else 1.0
    return 6.0 * rough * (area + lone * 4 * math.pi * reach ** 2) / (g * g)


def _room(case):
    return 20000 + 2 * int(_mesh_size(case))


def work(case):
    """Bytes: particles in (16 a particle, 12 without densities), positions and normals out (24 a mesh vertex, and
    indices), gradients out.  Flops: the pairs that contribute to a sum.  Mesh and band sizes come from the scenes'
    geometry and lie within about a third of the counted ones."""
    if case["use"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    n, method, use = case["n"], case["method"], case["use"]
    s, h, r, g, area, lone = _geometry(case)
    reach = _params(method, case["settings"])[4]
    verts = _mesh_size(case)
    ball = 4.0 / 3.0 * math.pi * (h / s) ** 3  # particles within h
    flops = 10.0 * area / (g * g) * 0.4 * ball * (33 if method == "yu13" else 16)
    if method == "yu13":
        flops += n * ball * reach ** 3 * (14 + 0.6 * 25)
    if method == "akinci12":
        flops += n * ball * 20
    if use == "indexed":
        return {"bytes": 12 * n + 24 * verts / 6 + 4 * verts, "flops": flops + n * ball * 10}
    if use == "train":  # the adjoint of every stage, the mesh's gradient in, the particles' out
        return {"bytes": 16 * n + 24 * verts + 12 * n, "flops": 2 * flops}
    return {"bytes": 16 * n + 24 * verts, "flops": flops}


# ------------------------------------------------------------------ 64 bits
# The public marching-cubes triangle table (Lorensen and Cline 1987, Bourke 1994): the cut edges of each of the 256
# cases in hexadecimal, three a triangle.  Bit i of a case: the field at corner i is at or below the iso value.
_TRI = (
    "- 083 019 183981 12a 08312a 92a029 2832a8a98 3b2 0b28b0 19023b 1b219b98b 3a1ba3 0a108a8ba 3903b9ba9 "
    "98aa8b 478 430734 019847 419471731 12a847 34730412a 92a902847 2a9297273794 8473b2 b47b24204 90184723b "
    "47b94b9b2921 3a13ba784 1ba14b1047b4 47890b9bab03 47b4b99ba 954 954083 054150 854835315 12a954 30812a495 "
    "52a542402 2a5325354348 95423b 0b208b495 05401523b 21525828b485 a3ba13954 4950818a18ba 54050b5bab03 "
    "54858aa8b 978579 930953573 078017157 153357 978957a12 a12950530573 802825857a52 2a5253357 7957893b2 "
    "95797292027b 23b018178157 b21b17715 958857a13a3b 5705097b010aba0 ba0b03a50807570 ba57b5 a65 0835a6 9015a6 "
    "1831985a6 165261 165126308 965906026 598582526328 23ba65 b08b20a65 01923b5a6 5a61929b298b 63b653513 "
    "08b0b50515b6 3b6036065059 65969bb98 5a6478 43047365a 1905a6847 a65197173794 612651478 125526304347 "
    "847905065026 739794329596269 3b2784a65 5a647242027b 01947823b5a6 9219b294b7b45a6 8473b53515b6 "
    "51b5b610b7b404b 059065036b63847 65969b4797b9 a4964a 4a649a083 a01a60640 83181686461a 149124264 "
    "308129249264 024426 832824426 a49a64b23 08228b49a4a6 3b201606461a 64161a48121b8b1 964936913b63 "
    "8b1810b61914641 3b6360064 648b68 7a678a89a 0730a709a67a a671a7178180 a67a71173 126168189867 "
    "269291679093739 780706602 732672 23ba68a89867 20727b09767a9a7 1801781a767a23b b21b17a61671 "
    "896867916b63136 091b67 7807063b0b60 7b6 76b 308b76 019b76 819831b76 a126b7 12a3086b7 2902a96b7 "
    "6b72a3a83a98 723627 708760620 276237019 162186198876 a76a17137 a7617a187108 03707a0a96a7 76a7a88a9 684b86 "
    "36b306046 86b846901 946963931b36 6846b82a1 12a30b06b046 4b846b0292a9 a93a32943b36463 823842462 042462 "
    "190234246438 194142246 8138618466a1 a10a06604 4634386a3039a93 a946a4 49576b 083495b76 50154076b "
    "b76834354315 954a1276b 6b712a083495 76b54a42a402 348354325a52b76 723762549 954086062687 362376150540 "
    "628687218485158 954a16176137 16a176107870954 40a4a503a6a737a 76a7a854a48a 6956b9b89 36b063056095 "
    "0b805b01556b 6b3635531 12a95b9b8b56 0b306b09656912a b85b56805a52025 6b36352a3a53 589528562382 956960062 "
    "158180568382628 156216 13616a386569896 a10a06950560 03856a a56 b5a75b b5ab75830 5b75ab190 a75ab7981831 "
    "b12b71751 08312717572b 9759279022b7 75272b592328982 25a235375 820852875a25 9015a35373a2 982921872a25752 "
    "135375 087071175 903935537 987597 5845a8ab8 5045b05abb30 01984a8aba45 ab4a45b34941314 2512852b8458 "
    "04b0b345b2b151b 0250592b5458b85 9452b3 25a352345384 5a2524420 3a235a385458019 5a2524192942 845853351 "
    "045105 845853905035 945 4b749b9ab 0834979b79ab 1ab1b414074b 3143481a474bab4 4b79b492b912 9749b791b2b1083 "
    "b74b42240 b74b42834324 29a279237749 9a7974a27870207 37a3a274a1a040a 1a2874 491417713 491417081871 403743 "
    "487 9a8ab8 30939bb9a 01a0a88ab 31ab3a 12b1b99b8 30939b1292b9 02b80b 32b 23828aa89 9a2092 23828a0181a8 1a2 "
    "138918 091 038 -"
).split()
_CORNER = ((0, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0), (1, 0, 0), (1, 0, 1), (1, 1, 1), (1, 1, 0))
_EDGE = ((0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7))
_SIGMA = 315.0 / (64.0 * math.pi)
MOST_CANDIDATES = 1.2e10  # of one frame: beyond, plain torch takes longer than a check should


def _params(method, settings):
    iso, ratio, scale, lam, reach = DEFAULTS[method]
    o = SETTINGS[method, settings]
    return (o.get("iso", iso), o.get("grid_ratio", ratio), o.get("cell_size_scale", scale),
            o.get("smoothing_lambda", lam), o.get("aniso_radius_over_h", reach))


class _Exact:
    """One frame in 64 bits."""

    def __init__(self, f, method, settings, own_density):
        self.dev = torch.device("cuda")
        f32 = np.float32
        iso, self.ratio, scale, self.lam, reach = _params(method, settings)
        self.method = method
        self.iso = float(f32(iso))
        self.h = float(f32(f.h))
        self.R = float(f32(f32(f.h) * f32(reach)))
        self.lam = float(f32(self.lam))
        self.rp, self.mass = float(f32(f.particle_radius)), float(f32(f.mass))
        self.cs = f32(f.h) * f32(scale)
        self.scs = self.cs / f32(self.ratio)
        lo = [f32(b) - self.cs for b in f.bbox_min]
        hi = [f32(b) + self.cs for b in f.bbox_max]
        self.min = [float(v) for v in lo]
        self.res = [int(f32((b - a) / self.cs) + f32(1)) for a, b in zip(lo, hi)]
        self.vres = [int(f32((b - a) / self.scs) + f32(1)) for a, b in zip(lo, hi)]
        x32 = torch.from_numpy(f.pos).to(self.dev)
        cell = self.cell_of(x32)
        key = self.key(cell)
        self.key_s, self.perm = torch.sort(key, stable=True)
        self.x32, self.cell = x32[self.perm], cell[self.perm]
        self.x = self.x32.double()
        C = self.res[0] * self.res[1] * self.res[2]
        count = torch.bincount(self.key_s, minlength=C)
        self.first = torch.zeros(C + 1, dtype=torch.int64, device=self.dev)
        self.first[1:] = count.cumsum(0)
        self.occ = (count > 0).view(self.res[2], self.res[1], self.res[0])
        rho = torch.from_numpy(f.density).to(self.dev).double()[self.perm]
        if own_density:
            c = math.ceil(self.h * 1.0001 / float(self.cs) + 1e-4)
            rho = torch.zeros_like(self.x[:, 0])
            for i, j, d in self.pairs(self.x, self.cell, c):
                u = 1 - d.square().sum(1) / self.h ** 2
                rho.index_add_(0, i, u.clamp(min=0) ** 3)
            rho *= self.mass * _SIGMA / self.h ** 3
        self.vol = self.mass / rho
        self.surface_and_band()

    def scalar(self, v):
        return torch.tensor(float(v), dtype=torch.float32, device=self.dev)

    def cell_of(self, p32):
        m = torch.tensor(self.min, dtype=torch.float32, device=self.dev)
        return ((p32 - m) / self.scalar(self.cs)).to(torch.int64)

    def key(self, c):
        return (c[:, 2] * self.res[1] + c[:, 1]) * self.res[0] + c[:, 0]

    def vertex(self, ids):
        """Index triples and 32-bit positions of grid vertices."""
        c = torch.stack([ids % self.vres[0], ids // self.vres[0] % self.vres[1],
                         ids // (self.vres[0] * self.vres[1])], 1)
        m = torch.tensor(self.min, dtype=torch.float32, device=self.dev)
        return c, (c.float() * self.scalar(self.scs)) + m

    def pairs(self, centres, cells, ext, most=1 << 27):
        """(i, j, x_j - centre_i) for the particles j of the cells within ext of each centre's, in chunks; rows of
        x-neighbouring cells are runs of the sorted particles."""
        r = torch.arange(-ext, ext + 1, device=self.dev)
        dz, dy = [v.reshape(-1) for v in torch.meshgrid(r, r, indexing="ij")]
        y, z = cells[:, 1:2] + dy, cells[:, 2:3] + dz
        ok = (y >= 0) & (y < self.res[1]) & (z >= 0) & (z < self.res[2])
        row = (z.clamp(0, self.res[2] - 1) * self.res[1] + y.clamp(0, self.res[1] - 1)) * self.res[0]
        x0 = (cells[:, 0:1] - ext).clamp(0, self.res[0] - 1)
        x1 = (cells[:, 0:1] + ext).clamp(0, self.res[0] - 1)
        beg = self.first[row + x0]
        num = torch.where(ok, self.first[row + x1 + 1] - beg, torch.zeros_like(beg))
        total = num.sum(1).cumsum(0)
        at, n = 0, centres.shape[0]
        while at < n:
            base = int(total[at - 1]) if at else 0
            to = max(at + 1, int(torch.searchsorted(total, base + most)))
            nn = num[at:to].reshape(-1)
            if int(nn.sum()):
                which = torch.repeat_interleave(torch.arange(nn.numel(), device=self.dev), nn)
                start = nn.cumsum(0) - nn
                j = beg[at:to].reshape(-1)[which] + torch.arange(which.numel(), device=self.dev) - start[which]
                i = at + which // dy.numel()
                yield i, j, self.x[j] - centres[i]
            at = to

    def near(self, cells):
        """Occupied cells within the clamped 3^3 and 5^3 boxes, as max pools."""
        return torch.nn.functional.max_pool3d(cells.float()[None, None], 5, 1, 2)[0, 0] > 0

    def surface_and_band(self):
        if self.method == "akinci12":
            grad = torch.zeros_like(self.x)
            nn = torch.zeros(len(self.x), device=self.dev)
            k = -45.0 / (math.pi * self.h ** 4)
            for i, j, d in self.pairs(self.x, self.cell, 1):
                dist = d.norm(dim=1)
                nn.index_add_(0, i, (dist > 0).float())
                w = torch.where((dist > 0) & (dist < self.h), k * (1 - dist / self.h).square() / dist, 0.0)
                grad.index_add_(0, i, (-(self.vol[j] * w))[:, None] * d)
            surface = (nn < 25) | (grad.norm(dim=1) > 3)
        else:
            empty = torch.nn.functional.max_pool3d((~self.occ).float()[None, None], 3, 1, 1)[0, 0] > 0
            s = self.occ & empty
            s[-1], s[:, -1], s[:, :, -1] = False, False, False
            surface = s.reshape(-1)[self.key_s]
            self.involved = (self.occ & self.near(s)).reshape(-1)[self.key_s]
        p = self.x32[surface]
        c = ((p - torch.tensor(self.min, dtype=torch.float32, device=self.dev)) / self.scalar(self.scs)).to(torch.int64)
        band = torch.zeros(self.vres[0] * self.vres[1] * self.vres[2], dtype=torch.bool, device=self.dev)
        reach = 1.5 * self.h
        m = self.min
        for oz in range(-3, 4):
            for oy in range(-3, 4):
                for ox in range(-3, 4):
                    v = c + torch.tensor([ox, oy, oz], device=self.dev)
                    ok = (v >= 0).all(1)
                    top = [torch.clamp(c[:, a] + 3, max=self.vres[a] - 1) for a in range(3)]
                    ok &= (v[:, 0] < top[0]) & (v[:, 1] <= top[1]) & (v[:, 2] <= top[2])
                    d = [v[:, a].float() * self.scalar(self.scs) + self.scalar(m[a]) - p[:, a] for a in range(3)]
                    dist = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
                    ok &= dist.double() < reach
                    w = v[ok]
                    band[(w[:, 2] * self.vres[1] + w[:, 1]) * self.vres[0] + w[:, 0]] = True
        self.band = band
        self.sv = band.nonzero()[:, 0]

    # -- smoothed particles and their matrices (as functions of the positions, for the gradient)
    def anisotropy(self, x):
        n = len(x)
        grad = x.requires_grad
        kept = list(self._close(x.detach(), x.detach(), 2, self.R, torch.arange(n, device=self.dev)))
        W = torch.zeros(n, dtype=torch.float64, device=self.dev)
        S = torch.zeros_like(self.x)
        for i, j in kept:
            w = 1 - _length(x[j] - x[i]) ** 3 / self.R ** 3
            W = W.index_add(0, i, w)
            S = S.index_add(0, i, w[:, None] * (x[j] - x[i]))
        mean = x + S / W[:, None]
        smooth = (1 - self.lam) * x + self.lam * mean
        del kept
        ids = self.involved.nonzero()[:, 0]
        at = torch.full((n,), -1, dtype=torch.int64, device=self.dev)
        at[ids] = torch.arange(len(ids), device=self.dev)
        A = torch.zeros(len(ids), 9, dtype=torch.float64, device=self.dev)
        Wc = torch.zeros(len(ids), dtype=torch.float64, device=self.dev)
        nn = torch.zeros(len(ids), dtype=torch.float64, device=self.dev)
        for i, j in self._close(mean.detach()[ids], x.detach(), 2, self.R, ids):
            v = x[j] - mean[ids[i]]
            w = 1 - _length(v) ** 3 / self.R ** 3
            nn.index_add_(0, i, torch.ones_like(w).detach())
            Wc = Wc.index_add(0, i, w)
            A = A.index_add(0, i, (w[:, None, None] * v[:, :, None] * v[:, None, :]).reshape(-1, 9))
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        lone = nn < MIN_NEIGHBORS
        C = (A.view(-1, 3, 3) + self.h ** 2 * eye) / torch.where(lone, 1.0, Wc)[:, None, None]
        C = torch.where(lone[:, None, None], torch.diag(torch.tensor([1.0, 2.0, 3.0], dtype=torch.float64,
                                                                     device=self.dev)), C)
        s, V = _eigen(C.detach())
        clamped = s[:, 0] < s[:, 2] / 4
        s = torch.maximum(s, s[:, 2:] / 4)
        G = (V / s[:, None, :]) @ V.transpose(1, 2) * (s.prod(1) ** (1.0 / 3.0) / self.h)[:, None, None]
        if grad:  # (1/h) cbrt(det C) C^-1 where no eigenvalue is clamped, else through the eigenvectors
            Gi = torch.linalg.inv(C) * (torch.linalg.det(C) ** (1.0 / 3.0) / self.h)[:, None, None]
            if bool(clamped.any()):
                q = clamped.nonzero()[:, 0]
                s, V = torch.linalg.eigh(C[q].cpu())
                s = torch.maximum(s, s[:, 2:] / 4)
                Gq = (V / s[:, None, :]) @ V.transpose(1, 2) * (s.prod(1) ** (1.0 / 3.0) / self.h)[:, None, None]
                Gi = Gi.index_copy(0, q, Gq.to(self.dev))
            G = Gi
        G = torch.where(lone[:, None, None], eye / self.h, G)
        return smooth, G, at

    def _close(self, centres, x, ext, r, owners):
        """Pairs within r, by chunks, from the windows about the owners' cells."""
        for i, j, d in self.pairs(centres, self.cell[owners], ext):
            ok = d.square().sum(1) < r * r
            yield i[ok], j[ok]

    # -- field values at the vertices `ids`
    def field(self, ids, x, rp, aniso=None):
        _, p32 = self.vertex(ids)
        v, cells = p32.double(), self.cell_of(p32)
        zero = torch.zeros(len(ids), dtype=torch.float64, device=self.dev)
        if self.method == "yu13":
            smooth, G, at = aniso
            c = _SIGMA * self.vol
            det = torch.linalg.det(G)
            phi = zero
            for i, j, _ in self.pairs(v, cells, 2, 1 << 26):
                with torch.no_grad():
                    inv = at[j] >= 0
                    d = smooth[j] - v[i]
                    q = d.square().sum(1)
                    if len(G):
                        q = torch.where(inv, _times(G[at[j].clamp(min=0)], d).square().sum(1), q)
                    ok = q < 1
                    i, j, inv = i[ok], j[ok], inv[ok]
                ii, jj = i[inv], j[inv]
                d = smooth[jj] - v[ii]
                q = _times(G[at[jj]], d).square().sum(1)
                phi = phi.index_add(0, ii, c[jj] * det[at[jj]] * (1 - q) ** 3)
                ii, jj = i[~inv], j[~inv]
                phi = phi.index_add(0, ii, c[jj] * (1 - (smooth[jj] - v[ii]).square().sum(1)) ** 3)
            return phi - 0.5
        h2 = self.h ** 2
        W, S = zero, torch.zeros(len(ids), 3, dtype=torch.float64, device=self.dev)
        for i, j, d in self.pairs(v, cells, 1):
            ok = d.square().sum(1) < h2
            i, j = i[ok], j[ok]
            d = x[j] - v[i]
            t = d.square().sum(1) / h2
            if self.method == "tc01":
                W = W.index_add(0, i, (t / 2) ** 2 - t / 2 + 0.25)
            else:
                w = (1 - t) ** 3
                W = W.index_add(0, i, w)
                S = S.index_add(0, i, w[:, None] * d)
        if self.method == "tc01":
            return W
        some = W > 0
        return torch.where(some, _length(S / torch.where(some, W, 1.0)[:, None]) - rp, 0.0)

    def mesh(self, phi):
        """Triangle soup: positions, normals, and what position_of() needs."""
        fill = float(np.array([0x64646464], np.uint32).view(np.float32)[0]) if self.method == "yu13" else 0.0
        rx, ry, rz = self.vres
        # with a border of zeros, one vertex below the grid and two above
        F = torch.zeros((rz + 3, ry + 3, rx + 3), dtype=torch.float64, device=self.dev)
        body = F[1:-2, 1:-2, 1:-2]
        body.fill_(fill)
        c, _ = self.vertex(self.sv)
        body[c[:, 2], c[:, 1], c[:, 0]] = phi
        inside = torch.zeros((rz + 1, ry + 1, rx + 1), dtype=torch.bool, device=self.dev)
        inside[:-1, :-1, :-1] = self.band.view(rz, ry, rx)
        corner = torch.tensor(_CORNER, device=self.dev)
        at = c[:, None, :] + corner  # (B, 8, 3)
        ok = inside[at[..., 2], at[..., 1], at[..., 0]].all(1)
        value = F[at[..., 2] + 1, at[..., 1] + 1, at[..., 0] + 1]
        self.margin = (value[ok] - self.iso).abs().min() if bool(ok.any()) else math.inf
        case = ((value <= self.iso) << torch.arange(8, device=self.dev)).sum(1)
        count = torch.tensor([0 if t == "-" else len(t) for t in _TRI], device=self.dev)
        edges = torch.tensor([[int(ch, 16) for ch in ("" if t == "-" else t).ljust(15, "0")] for t in _TRI],
                             device=self.dev)
        cube = (ok & (count[case] > 0)).nonzero()[:, 0]
        num = count[case[cube]]
        q = torch.repeat_interleave(torch.arange(len(cube), device=self.dev), num)
        k = torch.arange(len(q), device=self.dev) - (num.cumsum(0) - num)[q]
        cube = cube[q]
        e = edges[case[cube], k]
        ends = torch.tensor(_EDGE, device=self.dev)[e]  # (M, 2)
        a, b = [at[cube, ends[:, s]] for s in (0, 1)]
        va, vb = [value[cube, ends[:, s]] for s in (0, 1)]
        self.ends = a, b
        f = self.fraction(va, vb)

        def normal(p):
            g = []
            for axis in range(3):
                step = torch.zeros(3, dtype=torch.int64, device=self.dev)
                step[axis] = 1
                lo, hi = p - step + 1, p + step + 1
                g.append(F[lo[:, 2], lo[:, 1], lo[:, 0]] - F[hi[:, 2], hi[:, 1], hi[:, 0]])
            return self.unit(torch.stack(g, 1))

        na, nb = normal(a), normal(b)
        nrm = self.unit(na + f[:, None] * (nb - na))
        sign = -1.0 if self.iso < 0 and self.method != "akinci12" else 1.0
        return self.lerp(a, b, f), sign * nrm

    def unit(self, n):
        s = n.square().sum(1, keepdim=True)
        if self.method == "akinci12":  # left alone when no longer than 1e-7
            return torch.where(s.sqrt() > 1e-7, n / s.sqrt(), n)
        # a square beyond 32-bit floats (a difference with the value off the band) scales the normal to 0
        return n * torch.where(s > 3.4028235e38, 0.0, 1 / s.sqrt())

    def fraction(self, va, vb):
        d = vb - va
        small = d.abs() < 1e-7
        return torch.where(small, 0.5, (self.iso - va) / torch.where(small, 1.0, d))

    def lerp(self, a, b, f):
        m = torch.tensor(self.min, dtype=torch.float32, device=self.dev)
        pa, pb = [(c.float() * self.scalar(self.scs) + m).double() for c in (a, b)]
        return pa + f[:, None] * (pb - pa)

    def forward(self):
        with torch.no_grad():
            x = self.x
            aniso = self.anisotropy(x) if self.method == "yu13" else None
            return self.mesh(self.field(self.sv, x, self.rp, aniso))

    def gradients(self):
        """dL/dx in the input's order and dL/d(radius) with the topology held, from the field at the cut edges' ends."""
        a, b = [(c[:, 2] * self.vres[1] + c[:, 1]) * self.vres[0] + c[:, 0] for c in self.ends]
        ids, where = torch.unique(torch.cat([a, b]), return_inverse=True)
        x = self.x.clone().requires_grad_(True)
        rp = torch.tensor(self.rp, dtype=torch.float64, device=self.dev, requires_grad=True)
        aniso = self.anisotropy(x) if self.method == "yu13" else None
        phi = self.field(ids, x, rp, aniso)
        f = self.fraction(phi[where[:len(a)]], phi[where[len(a):]])
        g = torch.autograd.grad(_loss(self.lerp(*self.ends, f)), (x, rp), allow_unused=True)
        out = torch.zeros_like(x)
        out[self.perm] = g[0]
        return out, g[1]

    def decided(self):
        """Whether every cube's corners lie further from the iso value than a field in 32 bits is off."""
        off = {"zb05": 3e-7 * self.h, "akinci12": 3e-7 * self.h, "tc01": 1e-7, "yu13": 2e-7}[self.method]
        return bool(self.margin > off)

    def candidates(self):
        band = len(self.sv)
        per = len(self.x) / max(1, int(self.occ.sum()))
        return per * (125 * (band + 2 * len(self.x)) if self.method == "yu13" else 27 * band)


def _times(G, d):
    return (G * d[:, None, :]).sum(2)


def _length(v):
    """|v| with a gradient of 0 at 0."""
    s = v.square().sum(1)
    return torch.where(s > 0, s, 1.0).sqrt() * (s > 0)


def _eigen(C):
    """Ascending eigenvalues and eigenvectors of symmetric 3x3 matrices by cyclic Jacobi rotations."""
    A, V = C.clone(), torch.eye(3, dtype=torch.float64, device=C.device).expand_as(C).clone()
    for _ in range(10):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            t = 0.5 * torch.atan2(2 * A[:, p, q], A[:, q, q] - A[:, p, p])
            cs, sn = t.cos()[:, None], t.sin()[:, None]
            for M in (A, V):
                u, w = M[:, :, p].clone(), M[:, :, q].clone()
                M[:, :, p], M[:, :, q] = cs * u - sn * w, sn * u + cs * w
            u, w = A[:, p, :].clone(), A[:, q, :].clone()
            A[:, p, :], A[:, q, :] = cs * u - sn * w, sn * u + cs * w
    s = torch.diagonal(A, dim1=1, dim2=2)
    s, order = s.sort(1)
    return s, torch.gather(V, 2, order[:, None, :].expand(-1, 3, -1))


def exact(case, seed):
    """run()'s outputs; None for a mesh whose topology 32-bit rounding decides, and for counts and indices."""
    use = case["use"]
    if case["n"] > 3000000:
        return None
    if use == "batch":
        out = []
        for c, (m, f) in zip(_batch_cases(case), _batch_frames(case, seed)):
            e = _Exact(f, m, case["settings"], False)
            if e.candidates() > MOST_CANDIDATES / 4:
                return None
            pos, nrm = e.forward()
            sure = e.decided()
            out.append([_padded(v, _room(c)) if sure else None for v in (pos, nrm)] + [None])
        return out
    room = _room(case)
    e = _Exact(_scene(case["scene"], case["n"], seed), case["method"], case["settings"], use == "indexed")
    if e.candidates() > MOST_CANDIDATES:
        return None
    pos, nrm = e.forward()
    sure = e.decided()
    if use == "train":
        g, gr = e.gradients()
        return [_padded(pos, room) if sure else None, g, None] + ([gr] if case["method"] == "zb05" else [])
    if not sure:
        return None
    if use == "indexed":  # the first of the soup's vertices on each grid edge, in order of first use
        a, b = e.ends
        low, axis = torch.minimum(a, b), (a != b).to(torch.int64).argmax(1)
        key = 3 * ((low[:, 2] * e.vres[1] + low[:, 1]) * e.vres[0] + low[:, 0]) + axis
        _, which = torch.unique(key, return_inverse=True)
        first = torch.full((int(which.max()) + 1,), len(key), dtype=torch.int64, device=key.device)
        first.scatter_reduce_(0, which, torch.arange(len(key), device=key.device), "amin")
        first = first.sort()[0]
        return [_padded(pos[first], room), _padded(nrm[first], room), None, None, None]
    return [_padded(pos, room), _padded(nrm, room), None]


def _padded(rows, room):
    return torch.cat([rows, rows.new_zeros(room - rows.shape[0], 3)])
