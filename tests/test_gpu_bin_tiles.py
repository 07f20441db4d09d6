"""Bin tiles (mappings 7 and 8) where their work is split: tiles cut into pieces
whose sums the last CTA adds, a single row, a last tile of one row, frame counts
around a group's 32 or 64, whole tiles of a 2D table, every way pixels are
staged (4-byte copies, 2-byte pixels at odd offsets, 8-byte ones), and words of
per-frame masks."""
import ctypes

import numpy as np
import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

SHAPE = (701, 899)  # an odd pixel count: every second frame starts off a word
GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, poni1=340.3 * 172e-6,
            poni2=460.7 * 172e-6, rot1=0.01, rot2=-0.02, wavelength=1e-10)
CODES = {"uint16": N.DG_U16, "uint32": N.DG_U32, "int32": N.DG_I32, "float32": N.DG_F32,
         "float64": N.DG_F64}
# A sum is FP32 over 32 pairs (33 roundings, and a product, a weight's and a pixel's
# rounding each), then FP64: 40 * 2^-24 of the sum of its terms' sizes.
SUM = 40 * 2.0 ** -24
# Uniform pixels lie within 1.8 of their own deviation of the mean, so the shifted
# moments are at most 4 + 3 variances: half of 7 * SUM, and the shift's rounding.
STD = 4 * SUM


def _frames(torch, n, dtype, seed, offset):
    """n random frames, the first at `offset` elements past an aligned address."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    px = SHAPE[0] * SHAPE[1]
    lo = -500 if dtype == "int32" else 0
    kind = {"uint16": torch.int16, "uint32": torch.int32}.get(dtype) or getattr(torch, dtype)
    buf = torch.empty(offset + n * px, dtype=kind, device="cuda")
    for k in range(n):
        buf[offset + k * px:offset + (k + 1) * px] = torch.randint(
            lo, 2000, (px,), generator=g, device="cuda")
    return buf[offset:].view(n, px)


def _launch(torch, plan, frames, dtype, flags, masks=None):
    n, nb = frames.shape[0], plan.n_points * max(1, plan.n_azimuthal)
    outs = [torch.empty(n, nb, dtype=torch.float64, device="cuda")
            if want else None for want in (True, flags & N.DG_ERRORS, flags & N.DG_AZIMUTHAL_STD)]
    p = [None if o is None else ctypes.c_void_p(o.data_ptr()) for o in outs]
    torch.cuda.synchronize()
    at = ctypes.c_void_p(frames.data_ptr())
    if masks is None:
        N.check(N.lib().dg_integrate_device(plan.handle, at, CODES[dtype], n, flags, *p, None))
    else:
        N.check(N.lib().dg_integrate_dynamic_device(
            plan.handle, at, CODES[dtype], n, ctypes.c_void_p(masks.data_ptr()),
            masks.shape[1], flags, p[0], p[1], None))
    torch.cuda.synchronize()
    return [o.cpu().numpy() for o in outs if o is not None]


def _sums(rp, terms):
    return np.add.reduceat(np.append(terms, 0.0), rp[:-1]) * (np.diff(rp) > 0)


@pytest.mark.parametrize("variant,dtype,frames,bins,azimuthal,offset", [
    (8, "uint32", 130, 50, 0, 0),
    (8, "uint32", 1, 1, 0, 0),
    (8, "uint32", 63, 17, 0, 0),
    (8, "int32", 65, 50, 0, 0),
    (8, "float32", 65, 50, 0, 0),
    (8, "uint16", 65, 50, 0, 1),
    (8, "float64", 64, 33, 0, 0),
    (8, "uint32", 64, 40, 12, 0),
    (7, "int32", 33, 50, 0, 0),
    (7, "float32", 31, 25, 0, 0),
    (7, "uint16", 40, 50, 0, 1),
    (7, "float64", 32, 1, 0, 0),
])
def test_tiles_match_the_oracle(oracle, variant, dtype, frames, bins, azimuthal, offset):
    import torch
    it = dg.Integrator.from_poni_dict(GEOM, method="pixel_split", polarization_factor=0.9)
    mask = (np.random.default_rng(1).random(SHAPE) < 0.05).astype(np.uint8)
    it.set_mask(mask)
    plan = (it.prepare_cuda2d(SHAPE, bins, azimuthal) if azimuthal else
            it.prepare_cuda1d(SHAPE, bins, keep_tables=True))
    plan.gather_variant = variant
    x = _frames(torch, frames, dtype, 3, offset)
    if dtype.startswith("float"):
        x[0, 320_000] = float("nan")
        x[0, 320_001] = float("inf")
    std = 0 if azimuthal else N.DG_AZIMUTHAL_STD
    got = _launch(torch, plan, x, dtype, N.DG_ERRORS | std)
    # any frame alone gives the batch's bits
    for k in {0, frames // 2, frames - 1}:
        for a, b in zip(_launch(torch, plan, x[k:k + 1], dtype, N.DG_ERRORS | std), got):
            assert a[0].tobytes() == b[k].tobytes()
    again = _launch(torch, plan, x, dtype, N.DG_ERRORS | std)
    assert all(a.tobytes() == b.tobytes() for a, b in zip(again, got))
    if azimuthal:
        plan.gather_variant = 0
        for a, b in zip(_launch(torch, plan, x, dtype, N.DG_ERRORS), got):
            assert np.all(np.abs(a - b) <= 2 * SUM * np.abs(a))
        return
    p = oracle.poni(**GEOM)
    table = oracle.compact(oracle.build_ps1d(p, *SHAPE, bins), mask)
    rp, col, w, _ = plan.export_table(0)
    assert np.array_equal(rp, table.row_ptr) and np.array_equal(col, table.col)
    table.w = w
    norm = oracle.centres(p, *SHAPE, polarization_factor=0.9)["norm"]
    plain = _launch(torch, plan, x, dtype, N.DG_ERRORS)
    for k in {0, frames // 2, frames - 1}:
        f = x[k].cpu().numpy().view(dtype).astype(np.float64)
        i, s, d = oracle.azimuthal_std(table, None, norm, f, np.maximum(f, 0.0))
        size = _sums(rp, w * np.abs(np.where(np.isfinite(f), f, 0.0))[col])
        den = _sums(rp, w * norm[col])
        ok = np.isfinite(d) & (den > 0)
        assert np.array_equal(np.isnan(got[2][k]), np.isnan(d))
        assert np.all(np.abs(got[0][k] - i)[ok] <= 1.2 * SUM * (size / den)[ok])
        assert np.all(np.abs(got[1][k] - s)[ok] <= SUM * s[ok])
        if dtype != "int32":  # its negative pixels lie outside the bound's assumption
            assert np.all(np.abs(got[2][k] - d)[ok] <= STD * d[ok])
        if np.all(np.isfinite(f)):
            assert np.all(np.abs(plain[0][k] * den - _sums(rp, w * f[col])) <= SUM * size)
            v = _sums(rp, w * w * np.maximum(f, 0.0)[col])
            assert np.all(np.abs(plain[1][k] * den - np.sqrt(v)) <= SUM * np.sqrt(v))


@pytest.mark.parametrize("dtype,frames,offset", [
    ("uint32", 1, 0), ("uint32", 65, 0), ("uint16", 64, 1), ("float64", 3, 0)])
def test_words_of_frame_masks(oracle, dtype, frames, offset):
    import torch
    bins = 50
    it = dg.Integrator.from_poni_dict(GEOM, method="pixel_split", polarization_factor=0.9)
    plan = it.prepare_cuda1d(SHAPE, bins, keep_tables=True)
    plan.gather_variant = 8
    x = _frames(torch, frames, dtype, 7, offset)
    g = torch.Generator(device="cuda").manual_seed(8)
    masks = (torch.rand(x.shape, generator=g, device="cuda") < 0.1).to(torch.uint8)
    masks[frames - 1] = 1  # nothing left of the last frame
    got = _launch(torch, plan, x, dtype, N.DG_ERRORS, masks)
    rp, col, w, _ = plan.export_table(0)
    norm = oracle.centres(oracle.poni(**GEOM), *SHAPE, polarization_factor=0.9)["norm"]
    assert np.all(got[0][frames - 1] == 0.0) and np.all(got[1][frames - 1] == 0.0)
    for k in {0, frames // 2} - {frames - 1}:
        f = x[k].cpu().numpy().view(dtype).astype(np.float64)
        live = w * (masks[k].cpu().numpy() == 0)[col]
        den = _sums(rp, live * norm[col])
        ref = _sums(rp, live * f[col]) / den
        # the frame's norm sum rounds as its signal does
        assert np.all(np.abs(got[0][k] - ref) <= 2 * SUM * ref)
        v = np.sqrt(_sums(rp, live * live * f[col])) / den
        assert np.all(np.abs(got[1][k] - v) <= 2 * SUM * v)
