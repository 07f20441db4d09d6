"""Timed cases of the framework: azimuthal integration as its users run it.

Kinds of case (field ``kind``):

few    One to a few frames already on the GPU, integrated as they arrive (a live
       view, a feedback loop): ``dg_integrate_device`` on a plan pinned to the
       few-frame lane mapping (row warps), so that results are reproducible.
batch  A scan's worth of frames on the GPU, 1D pixel splitting:
       ``dg_integrate_device`` on a plan pinned to the batch lane mapping (bin
       tiles, two frames per lane), which the autotuner picks for such batches.
tuned  A batch of 2-byte supersampled frames, 1D or a 2D cake, on a plan whose
       lane mapping the autotuner chose, as a program does that runs long.
masks  Frames that each bring their own mask (dynamic masking):
       ``dg_integrate_dynamic_device``.
arrays A list of NumPy frames through ``Integrator.batch1d``, untuned: the plain
       Python call, host memory in and out.
bslz4  Bitshuffle/LZ4 chunks as they lie in a detector's HDF5 files, in host
       memory: ``Cuda1dPlan.integrate_bslz4_stack``.
first  A new geometry (recalibration, a moved detector): table construction and
       the first frame, ``Integrator.integrate1d`` on a fresh integrator.

Frames are seeded Poisson samples of powder rings on a background, with the
value ranges of the detector type; masks hold module gaps, 2% dead pixels and a
beam stop. ``exact`` computes the same results in 64 bits with plain torch: the
table by its own closed-form area integrals (pixel splitting) or by counting
samples (supersampling), the sums as sparse matrix products.
"""
import concurrent.futures
import ctypes
import math

import numpy as np
import torch

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

FEW_MAPPING, BATCH_MAPPING = 10, 8
CODES = {"uint16": N.DG_U16, "uint32": N.DG_U32, "int32": N.DG_I32, "float32": N.DG_F32}


# ----------------------------------------------------------------- the cases

def listed():
    eiger4m = dict(dim1=2167, dim2=2070, method="pixel_split", n_azimuthal=0)
    eiger9m = dict(dim1=3269, dim2=3110, method="supersampled", dtype="uint16", std=False)
    return [
        # A region of interest or a small detector, one frame: latency and launches.
        dict(name="roi_frame", kind="few", dim1=96, dim2=128, dtype="uint32", frames=1,
             method="pixel_split", bins=150, n_azimuthal=0, errors=True, std=False),
        # Live view of a 4M detector with error bars and azimuthal spread.
        dict(name="live_frame_4m", kind="few", dtype="uint32", frames=1, bins=2000, errors=True,
             std=True, **eiger4m),
        # Live cake of a 9M detector.
        dict(name="live_frame_cake", kind="few", frames=1, bins=1000, n_azimuthal=360,
             errors=True, **eiger9m),
        # A short series from a 300K detector through the plain Python call, odd sizes.
        dict(name="python_batch1d", kind="arrays", dim1=619, dim2=487, dtype="int32", frames=16,
             method="pixel_split", bins=700, n_azimuthal=0, errors=True, std=False),
        # A scan on a 1M detector with error bars.
        dict(name="pilatus_batch", kind="batch", dim1=1043, dim2=981, dtype="int32", frames=256,
             method="pixel_split", bins=1250, n_azimuthal=0, errors=True, std=False),
        # The benchmark's default workload: 4M detector, error bars and spread.
        dict(name="eiger4m_batch", kind="batch", dtype="uint32", frames=256, bins=2000,
             errors=True, std=True, **eiger4m),
        # Flat-field corrected frames: 32-bit floats, fine bins.
        dict(name="eiger4m_f32", kind="batch", dtype="float32", frames=128, bins=3000,
             errors=True, std=True, **eiger4m),
        # 9M detector, 16-bit frames, intensities only.
        dict(name="eiger9m_1d", kind="tuned", frames=64, bins=1000, n_azimuthal=0, errors=False,
             **eiger9m),
        # The same frames as 2D cakes with error bars.
        dict(name="eiger9m_cake", kind="tuned", frames=64, bins=1000, n_azimuthal=360,
             errors=True, **eiger9m),
        # Per-frame masks (diamond spots, cosmics) on the 4M detector.
        dict(name="eiger4m_masks", kind="masks", dtype="uint32", frames=64, bins=2000,
             errors=True, std=False, **eiger4m),
        # Compressed frames from a file, 1M detector.
        dict(name="pilatus_bslz4", kind="bslz4", dim1=1043, dim2=981, dtype="uint32", frames=16,
             method="pixel_split", bins=1250, n_azimuthal=0, errors=True, std=False),
        # Recalibration: a new table and its first frame.
        dict(name="new_geometry", kind="first", dim1=1043, dim2=981, dtype="int32", frames=1,
             method="pixel_split", bins=1250, n_azimuthal=0, errors=True, std=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["few", "few", "batch", "batch", "batch", "tuned", "masks", "arrays",
                       "bslz4", "first"])
    method, n_azimuthal, std = "pixel_split", 0, False
    errors = rng.random() < 0.75
    if kind == "few":
        dim1, dim2 = _log(rng, 96, 2167), _log(rng, 96, 2070)
        dtype, frames, bins = rng.choice(list(CODES)), rng.choice([1, 1, 2, 3, 4]), _log(rng, 100, 3000)
        std = rng.random() < 0.5
    elif kind == "batch":
        dim1, dim2 = _log(rng, 619, 2167), _log(rng, 619, 2070)
        dtype, frames, bins = rng.choice(["uint32", "int32", "float32"]), _log(rng, 48, 256), _log(rng, 800, 3000)
        std = rng.random() < 0.5
    elif kind == "tuned":
        method, dtype = "supersampled", "uint16"
        dim1, dim2 = _log(rng, 1043, 3269), _log(rng, 981, 3110)
        frames, bins = _log(rng, 16, 64), _log(rng, 500, 1000)
        n_azimuthal = rng.choice([0, 90, 180, 360])
    elif kind == "masks":
        dim1, dim2 = _log(rng, 1043, 2167), _log(rng, 981, 2070)
        dtype, frames, bins = rng.choice(["uint32", "int32"]), _log(rng, 24, 64), _log(rng, 800, 2000)
    elif kind == "arrays":
        dim1, dim2 = _log(rng, 96, 619), _log(rng, 96, 619)
        dtype, frames, bins = rng.choice(list(CODES)), rng.randint(2, 16), _log(rng, 150, 1000)
    elif kind == "bslz4":
        dim1, dim2 = _log(rng, 195, 1043), _log(rng, 487, 981)
        dtype, frames, bins = rng.choice(["uint16", "uint32", "int32"]), rng.randint(2, 16), _log(rng, 300, 1250)
    else:
        dim1, dim2 = _log(rng, 195, 1043), _log(rng, 487, 981)
        dtype, frames, bins = rng.choice(["uint32", "int32"]), 1, _log(rng, 300, 1250)
    return dict(kind=kind, dim1=dim1, dim2=dim2, dtype=dtype, frames=frames, method=method,
                bins=bins, n_azimuthal=n_azimuthal, errors=errors, std=std)


# ------------------------------------------------------- geometry and inputs

def _poni(c, seed):
    """Detector geometry: the beam near the middle for pixel splitting, near an
    edge for the supersampled workloads; another one for each seed of `first`."""
    px = 172e-6 if c["dim1"] * c["dim2"] < 2_000_000 else 75e-6
    edge = c["method"] == "supersampled"
    p = dict(pixel1=px, pixel2=px, distance=0.95 * c["dim1"] * px,
             poni1=(0.5 if edge else 0.52) * c["dim1"] * px,
             poni2=(0.013 if edge else 0.488) * c["dim2"] * px,
             rot1=0.05 if edge else 0.02, rot2=0.0 if edge else -0.01, rot3=0.0,
             wavelength=0.3e-10)
    if c["kind"] == "first":
        r = np.random.default_rng(seed)
        p["distance"] *= 1.0 + 0.02 * r.random()
        p["poni1"] += px * (r.random() - 0.5)
        p["poni2"] += px * (r.random() - 0.5)
    return p


def _trig(p):
    return (math.sin(p["rot1"]), math.cos(p["rot1"]), math.sin(p["rot2"]), math.cos(p["rot2"]),
            math.sin(p["rot3"]), math.cos(p["rot3"]))


def _angles(p, d1, d2):
    """2-theta and azimuth at detector positions d1, d2 (pixel units)."""
    s1, c1, s2, c2, s3, c3 = _trig(p)
    a, b, dist = d1 * p["pixel1"] - p["poni1"], d2 * p["pixel2"] - p["poni2"], p["distance"]
    x = a * c2 * c3 + b * (c3 * s1 * s2 - c1 * s3) - dist * (c1 * c3 * s2 + s1 * s3)
    y = a * c2 * s3 + b * (c1 * c3 + s1 * s2 * s3) - dist * (-(c3 * s1) + c1 * s2 * s3)
    z = a * s2 - b * c2 * s1 + dist * c1 * c2
    return torch.atan2(torch.sqrt(y * y + x * x), z), torch.atan2(x, y)


def _grid(n1, n2, off=0.5):
    d1 = torch.arange(n1, dtype=torch.float64, device="cuda")[:, None] + off
    d2 = torch.arange(n2, dtype=torch.float64, device="cuda")[None, :] + off
    return d1.expand(n1, n2), d2.expand(n1, n2)


def _mask(c, p):
    """Module gaps, 2% dead pixels and a beam stop; True where masked."""
    d1, d2 = c["dim1"], c["dim2"]
    m = torch.zeros(d1, d2, dtype=torch.bool)
    if d1 > 300:  # modules of 195 x 487 pixels, gaps of 17 x 7
        r, q = torch.arange(d1), torch.arange(d2)
        m |= (r % 212 >= 195)[:, None] | (q % 494 >= 487)[None, :]
    m |= torch.rand(d1, d2, generator=torch.Generator().manual_seed(7)) < 0.02
    if c["method"] == "pixel_split":
        # the beam: the pixel of the smallest scattering angle
        at = int(_angles(p, *_grid(d1, d2))[0].argmin())
        y, x = torch.arange(d1)[:, None] - at // d2, torch.arange(d2)[None, :] - at % d2
        m |= x * x + y * y < 6.0 ** 2
    return m.cuda()


def _frames(c, p, mask, seed):
    """Seeded frames on the GPU: rings on a background, Poisson-distributed;
    32-bit floats: 1e6 with 1e-3 relative noise (flat-field corrected)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = np.random.default_rng(seed)
    tth = torch.rad2deg(_angles(p, *_grid(c["dim1"], c["dim2"]))[0])
    bg, lo, hi = {"uint16": (200.0, 200.0, 2000.0), "uint32": (1e4, 500.0, 5000.0),
                  "int32": (50.0, 200.0, 5000.0), "float32": (1e6, 50.0, 200.0)}[c["dtype"]]
    lam = torch.full_like(tth, bg)
    for at, amp in zip(r.uniform(2.0, 30.0, 16), np.exp(r.uniform(np.log(lo), np.log(hi), 16))):
        lam += amp * torch.exp(-0.5 * ((tth - at) / 0.0212) ** 2)
    lam = lam.float()
    shape = (c["frames"], c["dim1"], c["dim2"])
    kind = {"uint16": torch.int16, "uint32": torch.int32, "int32": torch.int32,
            "float32": torch.float32}[c["dtype"]]
    out = torch.empty(shape, dtype=kind, device="cuda")
    for k in range(c["frames"]):
        if c["dtype"] == "float32":
            out[k] = lam * (1.0 + 1e-3 * torch.randn(lam.shape, generator=g, device="cuda"))
        else:
            out[k] = torch.poisson(lam, generator=g).to(kind)
            if c["dtype"] == "int32":
                out[k].masked_fill_(mask, -1)
    return {"uint16": lambda t: t.view(torch.uint16), "uint32": lambda t: t.view(torch.uint32)}.get(
        c["dtype"], lambda t: t)(out)


def _frame_masks(c, mask, seed):
    """Per-frame masks: the detector's own plus 1% of the pixels at random."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    out = torch.empty((c["frames"],) + tuple(mask.shape), dtype=torch.uint8, device="cuda")
    for k in range(c["frames"]):
        out[k] = mask | (torch.rand(mask.shape, generator=g, device="cuda") < 0.01)
    return out


def _integrator(c, p):
    return dg.Integrator.from_poni_dict(p, method=c["method"],
                                        n_ss=4 if c["method"] == "supersampled" else None,
                                        polarization_factor=0.99)


def _plan(c, it, n_frames, frames=None):
    shape = (c["dim1"], c["dim2"])
    if c["n_azimuthal"]:
        plan = it.prepare_cuda2d(shape, c["bins"], c["n_azimuthal"],
                                 azimuthal_range=(-math.pi, math.pi))
    else:
        plan = it.prepare_cuda1d(shape, c["bins"])
    if c["kind"] == "few":
        plan.gather_variant = FEW_MAPPING
    elif c["kind"] in ("batch", "masks"):
        plan.gather_variant = BATCH_MAPPING
    elif c["kind"] == "tuned":
        plan.autotune(frames, errors=c["errors"], azimuthal_std=c["std"])
    return plan


def prepare(case, seed):
    c = case
    p = _poni(c, seed)
    mask = _mask(c, p)
    frames = _frames(c, p, mask, seed)
    it = _integrator(c, p)
    s = dict(case=c)
    if c["kind"] == "masks":  # the frames' masks are complete; the plan has none
        s["masks"] = _frame_masks(c, mask, seed)
    else:
        it.set_mask(mask.cpu().numpy())
    if c["kind"] == "first":
        return dict(s, poni=p, mask=mask.cpu().numpy(), frame=frames[0].cpu().numpy())
    if c["kind"] == "arrays":
        host = frames.cpu().numpy()
        return dict(s, integrator=it, arrays=[np.ascontiguousarray(f) for f in host])
    if c["kind"] == "bslz4":
        host = frames.cpu().numpy()
        with concurrent.futures.ThreadPoolExecutor(8) as pool:
            s["chunks"] = list(pool.map(dg.bslz4_compress, host))
        return dict(s, plan=_plan(c, it, c["frames"]))
    plan = _plan(c, it, c["frames"], frames)
    n = c["bins"] * max(1, c["n_azimuthal"])
    outs = [torch.empty(c["frames"], n, dtype=torch.float64, device="cuda") if want else None
            for want in (True, c["errors"], c["std"])]
    return dict(s, plan=plan, frames=frames, outs=outs)


# ------------------------------------------------------------------ one pass

_stream = None


def _on_stream():
    """The program's own stream: every pass goes to it in order."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return ctypes.c_void_p(_stream.cuda_stream)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def run(state):
    s, c = state, state["case"]
    flags = (N.DG_ERRORS if c["errors"] else 0) | (N.DG_AZIMUTHAL_STD if c["std"] else 0)
    if c["kind"] == "first":
        it = _integrator(c, s["poni"])
        it.set_mask(s["mask"])
        r = it.integrate1d(s["frame"], c["bins"], c["errors"])
        return [r.intensity_array] + ([r.errors_array] if c["errors"] else [])
    if c["kind"] == "arrays":
        got = s["integrator"].batch1d(s["arrays"], c["bins"], c["errors"])
        return [[r.result.intensity_array for r in got]] + (
            [[r.result.errors_array for r in got]] if c["errors"] else [])
    if c["kind"] == "bslz4":
        return [o for o in s["plan"].integrate_bslz4_stack(s["chunks"], c["dtype"], c["errors"])
                if o is not None]
    oi, os_, od = s["outs"]
    stream = _on_stream()
    if c["kind"] == "masks":
        N.check(N.lib().dg_integrate_dynamic_device(
            s["plan"].handle, _ptr(s["frames"]), CODES[c["dtype"]], c["frames"], _ptr(s["masks"]),
            c["dim1"] * c["dim2"], flags, _ptr(oi), _ptr(os_), stream))
    else:
        N.check(N.lib().dg_integrate_device(s["plan"].handle, _ptr(s["frames"]),
                                            CODES[c["dtype"]], c["frames"], flags, _ptr(oi),
                                            _ptr(os_), _ptr(od), stream))
    return [o for o in (oi, os_, od) if o is not None]


# ------------------------------------------------------- what a pass must do

def work(case):
    """Frames (and masks) in, results out, the table once: 8 bytes an entry,
    about 2.6 (pixel splitting) or 2 entries a pixel; a multiply-add per entry,
    frame and sum. `bslz4` counts the decoded frames."""
    c = case
    px = c["dim1"] * c["dim2"]
    entries = (2.6 if c["method"] == "pixel_split" else 2.0) * px
    n = c["bins"] * max(1, c["n_azimuthal"])
    size = {"uint16": 2}.get(c["dtype"], 4) + (1 if c["kind"] == "masks" else 0)
    sums = 1 + (1 if c["errors"] else 0) + (2 if c["std"] else 0) + (1 if c["kind"] == "masks" else 0)
    outs = 1 + (1 if c["errors"] else 0) + (1 if c["std"] else 0)
    table = 2 * 8 * entries if c["kind"] == "first" else 8 * entries  # written, then read
    return {"bytes": c["frames"] * (px * size + n * outs * 8.0) + table,
            "flops": 2.0 * entries * c["frames"] * sums}


# ------------------------------------------------------------------- exact()

def _split_table(c, p):
    """Pixel splitting: (row, pixel, weight) of every pixel's quadrilateral in
    (2-theta, azimuth), cut at the bin edges. The area left of an edge is the
    boundary integral of azimuth d(2-theta) up to it."""
    d1, d2 = c["dim1"], c["dim2"]
    tth, chi = _angles(p, *_grid(d1 + 1, d2 + 1, 0.0))
    centre = _angles(p, *_grid(d1, d2))[1]
    lo, hi = tth.min().item(), tth.max().item() + 10.0 * 2.0 ** -52
    step = (hi - lo) / c["bins"]
    corners = [(slice(0, -1), slice(0, -1)), (slice(0, -1), slice(1, None)),
               (slice(1, None), slice(1, None)), (slice(1, None), slice(0, -1))]
    xs = [tth[i, j].reshape(-1) for i, j in corners]
    ys = []
    for i, j in corners:  # azimuth relative to the pixel's centre, unwrapped
        d = chi[i, j] - centre
        ys.append((d - 2 * math.pi * torch.round(d / (2 * math.pi))).reshape(-1))

    def left_of(e):
        total = torch.zeros_like(xs[0])
        for k in range(4):
            x0, y0, x1, y1 = xs[k], ys[k], xs[(k + 1) % 4], ys[(k + 1) % 4]
            slope = torch.where(x1 != x0, (y1 - y0) / (x1 - x0), torch.zeros_like(x0))
            a, b = torch.minimum(x0, e), torch.minimum(x1, e)
            total += (b - a) * 0.5 * (2 * y0 + slope * ((a - x0) + (b - x0)))
        return total

    x = torch.stack(xs)
    first = torch.floor((x.min(0).values - lo) / step).long()
    last = torch.floor((x.max(0).values - lo) / step).long().clamp(max=c["bins"] - 1)
    whole = left_of(x.max(0).values)
    rows, cols, weights = [], [], []
    left = torch.zeros_like(whole)
    # a pixel at the beam covers many bins; the beam stop masks it
    for k in range(min(64, int((last - first).max()) + 1)):
        right = left_of(lo + (first + k + 1).double() * step)
        w = ((right - left) / whole).abs()
        at = torch.nonzero((first + k <= last) & (w > 0)).reshape(-1)
        rows.append((first + k)[at])
        cols.append(at)
        weights.append(w[at])
        left = right
    return torch.cat(rows), torch.cat(cols), torch.cat(weights)


def _sample_table(c, p):
    """Supersampling: 4 x 4 samples a pixel, counted per bin."""
    d1, d2, ss = c["dim1"], c["dim2"], 4
    o = [(i + 0.5) / ss for i in range(ss)]
    y, x = _grid(d1, d2, 0.0)
    edge = [_angles(p, *_grid(d1, d2))[0]]
    along1 = (torch.arange(d1 * ss, dtype=torch.float64, device="cuda") + 0.5) / ss
    along2 = (torch.arange(d2 * ss, dtype=torch.float64, device="cuda") + 0.5) / ss
    for k in (o[0], d2 - o[0]):
        edge.append(_angles(p, along1, torch.full_like(along1, k))[0])
    for k in (o[0], d1 - o[0]):
        edge.append(_angles(p, torch.full_like(along2, k), along2)[0])
    r0 = min(e.min().item() for e in edge)
    r1 = max(e.max().item() for e in edge) + 3.0 * 2.0 ** -52
    dr, da = (r1 - r0) / c["bins"], 2 * math.pi / max(1, c["n_azimuthal"])
    pixel = torch.arange(d1 * d2, device="cuda").reshape(d1, d2)
    keys = []
    for i in o:
        for j in o:
            tth, chi = _angles(p, y + i, x + j)
            b = ((tth - r0) / dr).clamp(min=0).long().clamp(max=c["bins"] - 1)
            if c["n_azimuthal"]:
                turn = torch.remainder(chi + math.pi, 2 * math.pi)
                b += (turn / da).long().clamp(max=c["n_azimuthal"] - 1) * c["bins"]
            keys.append((b * (d1 * d2) + pixel).reshape(-1))
    keys, counts = torch.unique(torch.cat(keys), return_counts=True)
    return keys // (d1 * d2), keys % (d1 * d2), counts.double() / (ss * ss)


def _norm(c, p):
    """Solid angle times polarisation at the pixel centres."""
    d1, d2 = _grid(c["dim1"], c["dim2"])
    tth, chi = _angles(p, d1, d2)
    a, b = d1 * p["pixel1"] - p["poni1"], d2 * p["pixel2"] - p["poni2"]
    solid = (p["distance"] / torch.sqrt(a * a + b * b + p["distance"] ** 2)) ** 3
    c2 = torch.cos(tth) ** 2
    return (solid * 0.5 * (1.0 + c2 - 0.99 * torch.cos(2.0 * chi) * (1.0 - c2))).reshape(-1)


def exact(case, seed):
    c = case
    p = _poni(c, seed)
    mask = _mask(c, p)
    frames = _frames(c, p, mask, seed).reshape(c["frames"], -1)
    masks = _frame_masks(c, mask, seed).reshape(c["frames"], -1) if c["kind"] == "masks" else None
    rows, cols, w = (_split_table if c["method"] == "pixel_split" else _sample_table)(c, p)
    if masks is None:
        keep = ~mask.reshape(-1)[cols]
        rows, cols, w = rows[keep], cols[keep], w[keep]
    order = torch.argsort(rows * (c["dim1"] * c["dim2"]) + cols)
    rows, cols, w = rows[order], cols[order], w[order]
    n, px = c["bins"] * max(1, c["n_azimuthal"]), c["dim1"] * c["dim2"]
    start = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    start[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    norm = _norm(c, p)

    def times(weights, x):  # (bins x pixels) by (pixels x frames)
        return torch.sparse_csr_tensor(start, cols, weights, size=(n, px)) @ x

    intensity, sigma, spread = [], [], []
    whole = times(w, norm[:, None])
    for f0 in range(0, c["frames"], 8):
        s = frames[f0:f0 + 8]
        s = (s.to(torch.int64) if not s.is_floating_point() else s).double().T.contiguous()
        den = whole
        if masks is not None:
            live = (masks[f0:f0 + 8] == 0).double().T.contiguous()
            s, den = s * live, times(w, norm[:, None] * live)
        some = den > 0
        safe = torch.where(some, den, torch.ones_like(den))
        intensity.append((times(w, s) / safe * some).T)
        if c["errors"]:
            sigma.append((torch.sqrt(times(w * w, s.clamp(min=0))) / safe * some).T)
        if c["std"]:  # about a shift near the mean, which leaves little to cancel
            shift = (s.median(0).values / norm.median())[None, :]
            t = s - shift * norm[:, None]
            first, second = times(w, t), times(w / norm[cols], t * t)
            var = (second - first * first / safe) / safe
            spread.append(torch.where(some, torch.sqrt(var.clamp(min=0)),
                                      torch.full_like(var, math.nan)).T)
    outs = [torch.cat(o).contiguous() for o in (intensity, sigma, spread) if o]
    if c["kind"] == "first":
        return [o[0] for o in outs]
    return [list(o) for o in outs] if c["kind"] == "arrays" else outs
