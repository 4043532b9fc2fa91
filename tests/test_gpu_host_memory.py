"""Meshes copied to host arrays of every kind: never written (fresh pages),
in use, not starting at a page, pinned, and too small; the bytes are the device
mesh's, and bytes past the mesh stay as they were."""
import ctypes
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("memory", ["fresh", "used", "odd", "pinned"])
@pytest.mark.parametrize("n_side", [6, 40])
def test_host_arrays_of_every_kind(n_side, memory):
    import torch
    from fluidsurfacereconstructiongpu_gb300 import _native as N
    from fluidsurfacereconstructiongpu_gb300 import api, synthetic
    fr = synthetic.lattice_cube(n_side, 0.012, seed=4, origin=(0.3, 0.3, 0.3))
    rec = api.Reconstructor("zb05", 0, grid_ratio=4)
    header = api.header_of(fr)
    nv = rec.reconstruct(torch.from_numpy(fr.pos).cuda(), torch.from_numpy(fr.density).cuda(), header)
    want = [t.cpu().numpy() for t in rec.mesh_tensors()]
    assert nv > 0

    keep = []

    def array():
        size = 12 * nv + 200
        if memory == "pinned":
            keep.append(torch.zeros(size, dtype=torch.uint8).pin_memory())
            return keep[-1].numpy()
        keep.append(mmap.mmap(-1, size + 1000))
        a = np.frombuffer(keep[-1], np.uint8)
        if memory == "used":
            a[:] = 0
        return a[100:100 + size] if memory == "odd" else a[:size]

    out = ctypes.c_uint64(0)
    density = np.ascontiguousarray(fr.density)
    for call in ("copy", "host", "host"):
        pos, nrm = array(), array()
        if call == "copy":
            st = N.lib.fsr_copy_mesh(rec._h, pos.ctypes.data, nrm.ctypes.data, nv, ctypes.byref(out))
        else:
            st = N.lib.fsr_reconstruct_host(rec._h, ctypes.byref(header), fr.pos.ctypes.data, density.ctypes.data,
                                            fr.pos.shape[0], pos.ctypes.data, nrm.ctypes.data, nv, ctypes.byref(out),
                                            None)
        assert st == 0 and out.value == nv
        for got, ref in zip((pos, nrm), want):
            assert got[:12 * nv].tobytes() == ref.tobytes()
            assert not got[12 * nv:].any()
    st = N.lib.fsr_reconstruct_host(rec._h, ctypes.byref(header), fr.pos.ctypes.data, density.ctypes.data,
                                    fr.pos.shape[0], pos.ctypes.data, nrm.ctypes.data, nv - 1, ctypes.byref(out), None)
    assert st == 7 and out.value == nv
    rec.close()
