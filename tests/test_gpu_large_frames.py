"""64-bit float frames of more than 2^29 pixels (4 GiB): bin tiles stage the pixels
at their own addresses. The table holds the far corner alone."""
import ctypes as C
import math

import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

# FP32 sums over 32 pairs, then FP64, of both mappings (positive pixels)
SUM = 40 * 2.0 ** -24


@pytest.mark.parametrize("variant", [7, 8])
def test_pixels_beyond_four_gib(variant):
    import torch
    side, px, dist, bins = 23200, 1e-5, 0.5, 20
    assert side * side > 2 ** 29 > (side - 100) * side
    it = dg.Integrator.from_poni_dict(
        dict(pixel1=px, pixel2=px, distance=dist, poni1=0.0, poni2=0.0, wavelength=1e-10),
        method="counting", unit="2th_rad",
        radial_range=tuple(math.atan(math.hypot(side - d, side - d) * px / dist) for d in (80, 10)))
    plan = it.prepare_cuda1d((side, side), bins, max_batch_bytes=8 << 30)
    rp, col, _, _ = plan.export_table(0)
    assert rp[-1] > 1000 and col.max() >= 2 ** 29
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(side * side, generator=g, device="cuda", dtype=torch.float64)
    got = []
    for v in (0, variant):
        plan.gather_variant = v
        out = torch.full((bins,), -1.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        N.check(N.lib().dg_integrate_device(plan.handle, C.c_void_p(x.data_ptr()), N.DG_F64, 1, 0,
                                            C.c_void_p(out.data_ptr()), None, None, None))
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    plan.close()
    assert (abs(got[1] - got[0]) <= 2 * SUM * got[0]).all()
