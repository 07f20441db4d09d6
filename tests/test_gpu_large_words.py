"""32-bit frames of more than 2^30 pixels (4 GiB) on plans pinned to bin tiles, whose
offsets of 4-byte pixels have 32 bits. The table holds the far corner alone."""
import ctypes as C
import math

import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

# a weight's and a product's rounding and FP32 sums over 32 pairs, then FP64 (positive
# pixels): no mapping rounds more often
SUM = 40 * 2.0 ** -24


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("call", ["plain", "noalloc", "raw", "masked"])
def test_words_beyond_four_gib(variant, call):
    import torch
    side, px, dist, bins = 32800, 1e-5, 0.5, 20
    assert side * side > 2 ** 30
    it = dg.Integrator.from_poni_dict(
        dict(pixel1=px, pixel2=px, distance=dist, poni1=0.0, poni2=0.0, wavelength=1e-10),
        method="counting", unit="2th_rad",
        radial_range=tuple(math.atan(math.hypot(side - d, side - d) * px / dist) for d in (40, 5)))
    plan = it.prepare_cuda1d((side, side), bins, max_batch_bytes=16 << 30)
    rp, col, _, _ = plan.export_table(0)
    assert rp[-1] > 1000 and col.max() >= 2 ** 30
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randint(1, 2000, (side * side,), generator=g, device="cuda", dtype=torch.int32)
    masks = torch.zeros(side * side, device="cuda", dtype=torch.uint8)
    got = []
    for v in (0, variant):
        plan.gather_variant = v
        outs = [torch.full((bins,), -1.0, dtype=torch.float64, device="cuda") for _ in range(4)]
        p = [C.c_void_p(o.data_ptr()) for o in outs]
        frames = C.c_void_p(x.data_ptr())
        torch.cuda.synchronize()
        if call in ("plain", "noalloc"):
            fn = N.lib().dg_integrate_device if call == "plain" else N.lib().dg_integrate_device_noalloc
            N.check(fn(plan.handle, frames, N.DG_U32, 1, N.DG_ERRORS, p[0], p[1], None, None))
        else:
            N.check(N.lib().dg_integrate_raw_device(
                plan.handle, frames, N.DG_U32, 1,
                C.c_void_p(masks.data_ptr()) if call == "masked" else None,
                side * side if call == "masked" else 0, N.DG_ERRORS, *p, None))
        torch.cuda.synchronize()
        got.append(torch.stack(outs).cpu().numpy())
    plan.close()
    assert (abs(got[1] - got[0]) <= 2 * SUM * abs(got[0])).all() and (got[0][0] > 0).all()
