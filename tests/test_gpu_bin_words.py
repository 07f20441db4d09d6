"""Bin tiles stage 2-byte pixels as the words that hold them: the sums of uint16
frames equal those of the same values in uint32 bit for bit, for frames that begin
in either half of a word, odd and even pixel counts, the first and the last pixel,
frames stored bottom row first, few frames and many."""
import ctypes as C

import numpy as np
import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, rot1=0.01, rot2=-0.02, wavelength=1e-10)


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape,bins,order", [
    ((701, 899), 50, "detector"), ((701, 899), 50, "flip_vertical"), ((160, 201), 300, "flip_vertical"),
    ((160, 200), 300, "detector"), ((3, 5), 2, "detector")])
def test_words_give_the_sums_of_32_bit_pixels(variant, offset, shape, bins, order):
    import torch
    it = dg.Integrator.from_poni_dict(
        dict(GEOM, poni1=0.5 * shape[0] * 172e-6, poni2=0.4 * shape[1] * 172e-6), method="pixel_split")
    plan = it.prepare_cuda1d(shape, bins, input_order=order)
    plan.gather_variant = variant
    px = shape[0] * shape[1]
    _, col, _, _ = plan.export_table(0)
    assert {0, px - 1} <= set(np.unique(col)[[0, -1]].tolist())
    g = torch.Generator(device="cuda").manual_seed(6)
    wide = torch.randint(0, 65536, (70, px), generator=g, device="cuda", dtype=torch.int32)
    buf = torch.empty(offset + 70 * px, dtype=torch.int16, device="cuda")
    buf[offset:] = wide.to(torch.int16).reshape(-1)
    half = buf[offset:]
    masks = (torch.rand(70, px, generator=g, device="cuda") < 0.1).to(torch.uint8)
    L = N.lib()

    def sums(kind, data, code, n):
        o = [torch.full((n, bins), -1.0, dtype=torch.float64, device="cuda") for _ in range(4)]
        p = [C.c_void_p(t.data_ptr()) for t in o]
        torch.cuda.synchronize()
        at = C.c_void_p(data.data_ptr())
        if kind == "masks":
            st = L.dg_integrate_dynamic_device(plan.handle, at, code, n, C.c_void_p(masks.data_ptr()), px,
                                               N.DG_ERRORS, p[0], p[1], None)
        elif kind == "raw":
            st = L.dg_integrate_raw_device(plan.handle, at, code, n, None, 0, N.DG_ERRORS, *p, None)
        else:
            st = L.dg_integrate_device(plan.handle, at, code, n, kind, p[0], p[1] if kind else None,
                                       p[2] if kind & N.DG_AZIMUTHAL_STD else None, None)
        N.check(st)
        torch.cuda.synchronize()
        return torch.stack(o).view(torch.int64)

    for kind in (0, N.DG_ERRORS, N.DG_ERRORS | N.DG_AZIMUTHAL_STD, "raw", "masks"):
        for n in (1, 9, 33, 70):
            assert torch.equal(sums(kind, half, N.DG_U16, n), sums(kind, wide, N.DG_U32, n)), (kind, n)
    plan.close()
