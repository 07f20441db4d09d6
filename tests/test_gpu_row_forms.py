"""The forms of the row-warp launch (few CTAs per SM, many, many of short rows, long
rows in groups) sum every row alike: each frame of a batch equals the frame alone,
bit for bit, and a mapping with FP32 partial sums to rounding."""
import ctypes as C

import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, rot1=0.01, rot2=-0.02, wavelength=1e-10)
CODES = {"uint16": N.DG_U16, "uint32": N.DG_U32, "float32": N.DG_F32, "float64": N.DG_F64}
SUM = 40 * 2.0 ** -24  # FP32 over 32 pairs and their roundings


def _launch(torch, plan, x, dtype, flags, bins):
    outs = [torch.full((x.shape[0], bins), -1.0, dtype=torch.float64, device="cuda")
            if want else None for want in (True, flags & N.DG_ERRORS, flags & N.DG_AZIMUTHAL_STD)]
    torch.cuda.synchronize()
    N.check(N.lib().dg_integrate_device(
        plan.handle, C.c_void_p(x.data_ptr()), CODES[dtype], x.shape[0], flags,
        *[None if o is None else C.c_void_p(o.data_ptr()) for o in outs], None))
    torch.cuda.synchronize()
    return [o for o in outs if o is not None]


@pytest.mark.parametrize("dtype", sorted(CODES))
@pytest.mark.parametrize("shape,bins,azimuthal", [
    ((300, 300), 100, 0),     # few CTAs per SM, for any number of frames
    ((619, 487), 1000, 0),    # many: long rows, and groups of them in larger batches
    ((619, 487), 500, 90),    # many: short rows
    ((1043, 981), 3000, 0),
])
def test_frames_of_a_batch_equal_frames_alone(shape, bins, azimuthal, dtype):
    import torch
    it = dg.Integrator.from_poni_dict(
        dict(GEOM, poni1=0.5 * shape[0] * 172e-6, poni2=0.4 * shape[1] * 172e-6),
        method="supersampled" if azimuthal else "pixel_split", n_ss=2 if azimuthal else None)
    plan = it.prepare_cuda2d(shape, bins, azimuthal) if azimuthal else it.prepare_cuda1d(shape, bins)
    n_bins, n = bins * max(1, azimuthal), 24
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randint(1, 2000, (n,) + shape, generator=g, device="cuda").to(
        {"uint16": torch.int16, "uint32": torch.int32}.get(dtype) or getattr(torch, dtype))
    for flags in (0, N.DG_ERRORS) + (() if azimuthal else (N.DG_ERRORS | N.DG_AZIMUTHAL_STD,)):
        plan.gather_variant = 0
        other = _launch(torch, plan, x[:4], dtype, flags, n_bins)
        plan.gather_variant = 10
        batch = _launch(torch, plan, x, dtype, flags, n_bins)
        for a, b in zip(batch[:2], other[:2]):
            assert bool(((a[:4] - b).abs() <= SUM * b.abs()).all())
        for count in (1, 2, 4, 7):
            part = _launch(torch, plan, x[:count], dtype, flags, n_bins)
            for a, b in zip(part, batch):
                assert torch.equal(a.view(torch.int64), b[:count].view(torch.int64))
    plan.close()
