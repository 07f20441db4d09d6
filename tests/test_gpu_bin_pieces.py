"""Bin tiles of tables whose small tiles are cut like their large neighbours (few
azimuthal sectors with a radial range, a beam near a corner, few inner pixels left
by a mask), against the entry-lane mapping: every result is written by every
launch."""
import ctypes
import math

import numpy as np
import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N
from test_bin_items import bin_items, check_items

pytestmark = pytest.mark.gpu

PX, DIST = 172e-6, 0.2
# both mappings' sums of positive pixels: FP32 over 32 pairs (33 roundings, and a
# product, a weight's and a pixel's rounding each), then FP64
SUM = 40 * 2.0 ** -24


def _plan(shape, beam, method, bins, azimuthal, radial_range, mask=None):
    it = dg.Integrator.from_poni_dict(
        dict(pixel1=PX, pixel2=PX, distance=DIST, poni1=beam[0] * PX, poni2=beam[1] * PX,
             wavelength=1e-10), method=method, radial_range=radial_range)
    if mask is not None:
        it.set_mask(mask)
    return it.prepare_cuda2d(shape, bins, azimuthal) if azimuthal else it.prepare_cuda1d(shape, bins)


def _launch(torch, plan, frames, n_bins):
    outs = [torch.full((frames.shape[0], n_bins), math.nan, dtype=torch.float64, device="cuda")
            for _ in range(2)]
    torch.cuda.synchronize()
    N.check(N.lib().dg_integrate_device(
        plan.handle, ctypes.c_void_p(frames.data_ptr()), N.DG_U32, frames.shape[0], N.DG_ERRORS,
        *[ctypes.c_void_p(o.data_ptr()) for o in outs], None, None))
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in outs]


def _compare(plan, variant, shape, n_bins, frames):
    import torch
    rp, col, _, _ = plan.export_table(0)
    assert check_items(bin_items(variant, rp, col), n_bins) > 1
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(1, 2000, (frames,) + shape, generator=g, device="cuda", dtype=torch.int32)
    plan.gather_variant = 0
    want = _launch(torch, plan, x, n_bins)
    plan.gather_variant = variant
    for _ in range(2):
        for a, b in zip(_launch(torch, plan, x, n_bins), want):
            assert np.array_equal(np.isnan(a), np.isnan(b))
            assert np.all(np.abs(a - b) <= 2 * SUM * np.abs(b))
    for a, b in zip(_launch(torch, plan, x[1:2], n_bins), want):  # one frame alone
        assert np.all(np.abs(a[0] - b[1]) <= 2 * SUM * np.abs(b[1]))
    plan.close()


@pytest.mark.parametrize("variant,shape,method,bins,azimuthal", [
    (8, (1043, 981), "pixel_split", 496, 4),
    (8, (1043, 981), "pixel_split", 368, 2),
    (8, (2167, 2070), "counting", 500, 8),
    (7, (2167, 2070), "counting", 1000, 4),
])
def test_few_sectors(variant, shape, method, bins, azimuthal):
    end = math.atan(0.48 * shape[1] * PX / DIST)
    plan = _plan(shape, (0.5 * shape[0], 0.5 * shape[1]), method, bins, azimuthal, (1e-4, end))
    _compare(plan, variant, shape, bins * azimuthal, 70)


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("shape,off,bins", [((701, 899), 10, 50), ((1043, 981), 60, 82)])
def test_beam_near_a_corner(variant, shape, off, bins):
    plan = _plan(shape, (off, off), "pixel_split", bins, 0, None)
    _compare(plan, variant, shape, bins, 65)


@pytest.mark.parametrize("variant", [7, 8])
@pytest.mark.parametrize("left", [0.002, 0.01])
def test_few_inner_pixels_left(variant, left):
    shape, bins = (1043, 981), 100
    rows = 24 if variant == 7 else 16
    whole = _plan(shape, (500.3, 500.3), "pixel_split", bins, 0, None)
    rp, col, _, _ = whole.export_table(0)
    whole.close()
    inner = np.unique(col[:rp[rows]])
    mask = np.zeros(shape, np.uint8)
    mask.ravel()[inner[np.random.default_rng(3).random(inner.size) >= left]] = 1
    plan = _plan(shape, (500.3, 500.3), "pixel_split", bins, 0, None, mask)
    _compare(plan, variant, shape, bins, 65)
