"""The pair kernels take the square root of a squared distance and divide by
the neighbour radius R with FMA corrections instead of the IEEE operations'
sequences; the root must be the correctly rounded one for every float of its
range, and the weight 1 - (d/R)^3 the IEEE one for every squared distance.
Radii outside [2^-20, 2^40] take the IEEE operations: a frame scaled by a power
of two (every FP32 operation scales exactly) must give the scaled mesh."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [0.016, 0.072, 1.0, 123.456, 7e-6, 2.0 ** -20, 2.0 ** 40])
def test_root_and_weight_match_ieee(R):
    import torch
    from fluidsurfacereconstructiongpu_gb300 import _native as N
    torch.cuda.init()
    checked, bad = ctypes.c_uint64(), ctypes.c_uint64()
    N.check(N.lib.fsr_check_root(float(np.float32(R)), ctypes.byref(checked), ctypes.byref(bad)))
    assert checked.value > 1.6e9
    assert bad.value == 0, (R, bad.value)


@pytest.mark.parametrize("shift", [-18, -14, 12])
def test_scaled_frames_give_scaled_means(shift):
    """h = 0.05: 2^-18 puts R below the fast range, 2^-14 and 2^12 inside."""
    import torch
    from fluidsurfacereconstructiongpu_gb300 import api, synthetic
    fr = synthetic.lattice_cube(12, 0.0125, seed=6, jitter_frac=0.4)
    s = 2.0 ** shift
    out = []
    for k in (1.0, s):
        rec = api.Reconstructor("yu13", 0)
        hd = api.header_from(fr.bbox_min * k, fr.bbox_max * k, fr.h * k, fr.particle_radius * k, fr.mass * k ** 3)
        rec.reconstruct(torch.from_numpy(fr.pos * np.float32(k)).cuda(), torch.from_numpy(fr.density).cuda(), hd)
        out.append(rec.debug("mean"))
        rec.close()
    assert np.array_equal(out[0] * np.float32(s), out[1])
