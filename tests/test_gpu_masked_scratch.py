"""Masked and raw calls on bin tiles reserve partial sums for the pieces of cut tiles
alone, not for the segments of the mappings that the call does not use."""
import ctypes as C

import numpy as np
import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,masked,sums", [(8, True, 4), (8, False, 2), (7, False, 2)])
def test_partial_sums_of_the_tiles(variant, masked, sums):
    import torch
    shape, bins, n = (1043, 981), 1250, 64
    it = dg.Integrator.from_poni_dict(
        dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, poni1=0.09, poni2=0.08, wavelength=1e-10),
        method="pixel_split")
    plan = it.prepare_cuda1d(shape, bins)
    rp, col, _, _ = plan.export_table(0)
    rp, col = np.ascontiguousarray(rp, np.int64), np.ascontiguousarray(col, np.int32)
    counts = np.zeros(5, np.int64)
    N.check(N.lib().dg_test_bin_items(variant, bins, rp.ctypes.data, col.ctypes.data,
                                      counts.ctypes.data, *[None] * 5))
    assert counts[4] > 0
    x = torch.ones((n,) + shape, dtype=torch.int32, device="cuda")
    masks = torch.zeros((n,) + shape, dtype=torch.uint8, device="cuda") if masked else None
    outs = [torch.empty((n, bins), dtype=torch.float64, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    plan.gather_variant = variant

    def held(frames):
        N.check(N.lib().dg_integrate_raw_device(
            plan.handle, C.c_void_p(x.data_ptr()), N.DG_U32, frames,
            C.c_void_p(masks.data_ptr()) if masked else None, shape[0] * shape[1] if masked else 0,
            N.DG_ERRORS, *[C.c_void_p(o.data_ptr()) for o in outs], None))
        torch.cuda.synchronize()
        return plan.info().device_bytes

    few = held(32)
    assert held(64) - few == counts[4] * sums * 32 * 8
    assert torch.equal(outs[0][0], outs[0][n - 1]) and bool((outs[0] > 0).any())
    plan.close()
