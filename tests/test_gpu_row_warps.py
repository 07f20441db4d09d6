"""Row warps (mapping 10): long rows by a CTA each and, in launches that fill the
chip, by groups of neighbours (with a last group of fewer), rows of a warp, rows
of eight lanes, and non-finite pixels at the ends of rows, where a row's last
entry is loaded again with weight 0."""
import numpy as np
import pytest

import dioptrin_b200 as dg

pytestmark = pytest.mark.gpu

SHAPE = (701, 899)
GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, poni1=340.3 * 172e-6,
            poni2=460.7 * 172e-6, rot1=0.01, rot2=-0.02, wavelength=1e-10)
# a weight rounds once to FP32 and the sums are FP64
SUM = 2.0 ** -23
# as above, through moments of at most 4 + 3 variances (pixels within 1.8 of their
# deviation of the mean) and the FP32 quotient c/n, halved by the root
STD = 16 * 2.0 ** -24


def _sums(rp, terms):
    return np.add.reduceat(np.append(terms, 0.0), rp[:-1]) * (np.diff(rp) > 0)


@pytest.mark.parametrize("bins,frames,dtype", [
    (1003, 22, "uint16"),    # groups of eight and one of three
    (1003, 22, "float32"),
    (1003, 4, "uint32"),     # a CTA per row
    (1003, 1, "int32"),
    (7, 3, "float64"),       # fewer long rows than a group
    (4001, 6, "uint16"),     # a warp per row
    (40009, 5, "float32"),   # eight lanes per row
    (40009, 1, "uint16"),
    (2600, 2, "float32"),    # rows on both sides of the longest kind's limit
])
def test_rows_match_the_oracle(oracle, bins, frames, dtype):
    rng = np.random.default_rng(bins + frames)
    it = dg.Integrator.from_poni_dict(GEOM, method="pixel_split", polarization_factor=0.9)
    mask = (rng.random(SHAPE) < 0.05).astype(np.uint8)
    it.set_mask(mask)
    plan = it.prepare_cuda1d(SHAPE, bins, keep_tables=True)
    plan.gather_variant = 10
    rp, col, w, _ = plan.export_table(0)
    x = rng.integers(-300 if dtype == "int32" else 0, 2000, (frames,) + SHAPE).astype(dtype)
    odd = dtype.startswith("float")
    if odd:  # the last entries' pixels of some rows, in the first frame
        ends = col[rp[1:][np.diff(rp) > 0][::97] - 1]
        x[0].ravel()[ends] = np.where(np.arange(ends.size) % 2, np.nan, np.inf)
    gi, gs, gd = plan.integrate_stack(x, True, True)
    pi, ps, _ = plan.integrate_stack(x, True)
    for k in range(frames):  # any frame alone gives the batch's bits
        si, ss, sd = plan.integrate_stack(x[k:k + 1], True, True)
        assert si[0].tobytes() == gi[k].tobytes() and ss[0].tobytes() == gs[k].tobytes()
        assert sd[0].tobytes() == gd[k].tobytes()
        si, ss, _ = plan.integrate_stack(x[k:k + 1], True)
        assert si[0].tobytes() == pi[k].tobytes() and ss[0].tobytes() == ps[k].tobytes()
    p = oracle.poni(**GEOM)
    table = oracle.compact(oracle.build_ps1d(p, *SHAPE, bins), mask)
    assert np.array_equal(rp, table.row_ptr) and np.array_equal(col, table.col)
    table.w = w
    norm = oracle.centres(p, *SHAPE, polarization_factor=0.9)["norm"]
    den = _sums(rp, w * norm[col])
    for k in {0, frames - 1}:
        f = x[k].ravel().astype(np.float64)
        i, s, d = oracle.azimuthal_std(table, None, norm, f, np.maximum(f, 0.0))
        assert np.array_equal(np.isnan(gd[k]), np.isnan(d))
        size = _sums(rp, w * np.abs(np.where(np.isfinite(f), f, 0.0))[col])
        ok = np.isfinite(d) & (den > 0)
        # where all pixels count (what is left of a row's weight after exclusions is a
        # difference, whose error the remainder does not bound)
        ok &= _sums(rp, (~np.isfinite(f)).astype(np.float64)[col]) == 0
        assert np.all(np.abs(gi[k] - i)[ok] <= 2 * SUM * (size / den)[ok])
        assert np.all(np.abs(gs[k] - s)[ok] <= 2 * SUM * s[ok])
        # rows of many entries: the bound on the moments is a statement about samples
        many = ok & (np.diff(rp) > 64) & (dtype != "int32")
        assert np.all(np.abs(gd[k] - d)[many] <= STD * d[many])
        ref = np.divide(_sums(rp, w * f[col]), den, out=np.zeros(bins), where=den > 0)
        assert np.array_equal(np.isnan(pi[k]), np.isnan(ref))
        assert np.array_equal(np.isinf(pi[k]), np.isinf(ref))
        fin = np.isfinite(ref)
        assert np.all(np.abs(pi[k][fin] - ref[fin]) * den[fin] <= SUM * size[fin])
        if not odd or k:
            v = np.sqrt(_sums(rp, w * w * np.maximum(f, 0.0)[col]))
            assert np.all(np.abs(ps[k] * den - v) <= SUM * v)
