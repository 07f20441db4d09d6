"""Partial sums of the bin tiles are kept for the pieces of cut tiles alone: a table
of one heavy tile and many small ones needs no room for the small ones."""
import numpy as np
import pytest

from dioptrin_b200 import _native as N


def _counts(variant, rp, col):
    counts = np.zeros(5, np.int64)
    N.check(N.lib().dg_test_bin_items(variant, len(rp) - 1, rp.ctypes.data, col.ctypes.data,
                                      counts.ctypes.data, *[None] * 5))
    return [int(v) for v in counts]


@pytest.mark.parametrize("variant", [7, 8])
def test_small_tiles_keep_none(variant):
    rng = np.random.default_rng(1)
    heavy = np.sort(rng.permutation(400_000).astype(np.int32).reshape(20, -1), axis=1)
    small = np.tile(np.arange(3, dtype=np.int32), 100_000)
    rp = np.concatenate([[0], np.cumsum([heavy.shape[1]] * 20 + [3] * 100_000)]).astype(np.int64)
    items, rows, tiles, _, partial = _counts(variant, rp, np.concatenate([heavy.ravel(), small]))
    pieces = items - tiles  # beyond one per tile: all of the few heavy tiles
    assert 1 <= pieces <= 400
    assert pieces + 1 <= partial // rows <= pieces + 4 and partial % rows == 0
    assert _counts(variant, rp[20:] - rp[20], small)[4] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [7, 8])
def test_many_empty_bins_fit_the_fixed_array(variant):
    """A radial range far beyond the detector: 720,000 bins, all but the first few
    hundred empty. Six sums for each would exceed the fixed 32 MiB for one frame."""
    import ctypes as C

    import dioptrin_b200 as dg
    import torch
    shape, bins, n = (1043, 981), 720_000, 3
    it = dg.Integrator.from_poni_dict(
        dict(pixel1=1e-4, pixel2=1e-4, distance=200.0, poni1=0.05, poni2=0.05, wavelength=1e-10),
        method="pixel_split", radial_range=(0.0, 1.5))
    plan = it.prepare_cuda1d(shape, bins)
    plan.gather_variant = variant
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.rand((n,) + shape, generator=g, device="cuda")
    got = []
    for fn in (N.lib().dg_integrate_device, N.lib().dg_integrate_device_noalloc):
        outs = [torch.full((n, bins), -1.0, dtype=torch.float64, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        N.check(fn(plan.handle, C.c_void_p(x.data_ptr()), N.DG_F32, n,
                   N.DG_ERRORS | N.DG_AZIMUTHAL_STD, *[C.c_void_p(o.data_ptr()) for o in outs], None))
        torch.cuda.synchronize()
        got.append([o.cpu().numpy() for o in outs])
    assert np.any(got[0][0] > 0) and np.all(got[0][0] >= 0)
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)
    plan.close()
