"""Per-row plan data against the oracle at the bin counts where the row kernels
change shape: rows of more than 256 entries on average take a CTA, shorter ones
a warp; a single row, rows without entries, and a beam pixel that covers more
bins than a fill thread buffers."""
import numpy as np
import pytest

import dioptrin_b200 as dg

pytestmark = pytest.mark.gpu

SHAPE = (96, 128)
GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.1, poni1=40.3 * 172e-6,
            poni2=60.7 * 172e-6, rot1=0.01, rot2=-0.02, wavelength=1e-10)


@pytest.mark.parametrize("bins", [1, 7, 100, 150, 8000])
def test_row_sums_and_tables_match_oracle(oracle, bins):
    rng = np.random.default_rng(5)
    mask = (rng.random(SHAPE) < 0.05).astype(np.uint8)
    it = dg.Integrator.from_poni_dict(GEOM, method="pixel_split", polarization_factor=0.9)
    it.set_mask(mask)
    plan = it.prepare_cuda1d(SHAPE, bins, keep_tables=True)
    p = oracle.poni(**GEOM)
    full = oracle.build_ps1d(p, *SHAPE, bins)
    rp, col, _, _ = plan.export_table(1)
    assert np.array_equal(rp, full.row_ptr) and np.array_equal(col, full.col)
    table = oracle.compact(full, mask)
    rp, col, w, den = plan.export_table(0)
    assert np.array_equal(rp, table.row_ptr) and np.array_equal(col, table.col)
    # the row sums are checked on the plan's own weights (their parity with the
    # oracle's is tested elsewhere)
    table.w = w
    norm = oracle.centres(p, *SHAPE, polarization_factor=0.9)["norm"]
    ref = oracle.denominators(table, norm)
    # two orders of adding n positive terms differ by at most 2 (n - 1) 2^-53,
    # and a term by the device's cos (a few ulp, 1e-14 allowed)
    tol = 2.0 * max(1, int(np.max(np.diff(rp)))) * 2.0 ** -53 + 1e-14
    assert np.all(np.abs(den - ref) <= tol * ref)
    frame = rng.poisson(500.0, SHAPE).astype(np.uint32)
    raw = plan.integrate1d_raw(frame)
    assert np.array_equal(raw.sum_norm, den)
    count = np.add.reduceat(np.append(table.w, 0.0), rp[:-1]) * (np.diff(rp) > 0)
    assert np.all(np.abs(raw.count - count) <= (tol + 2e-9) * np.maximum(count, 1e-3))
    # origin and validity counts: a one-entry bin has no spread, an empty one none at all
    plan.gather_variant = 10
    got = plan.integrate1d(frame, errors=True, azimuthal_std=True)
    i, s, d = oracle.azimuthal_std(table, None, norm, frame.ravel().astype(np.float64),
                                   frame.ravel().astype(np.float64))
    for a, b in ((got.intensity_array, i), (got.errors_array, s), (got.azimuthal_std_array, d)):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        ok = ~np.isnan(b)
        assert np.all(np.abs(a[ok] - b[ok]) <= 1e-5 * np.maximum(np.abs(b[ok]), 1.0))
