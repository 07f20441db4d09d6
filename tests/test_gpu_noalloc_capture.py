"""The allocation-free call under stream capture: after a warm-up on the plan's
stream it is captured on another one, replayed on new frames, and replayed beside
plain calls of the same plan on a third stream; each agrees with the plain call
bit for bit."""
import ctypes as C

import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.2, poni1=80.3 * 172e-6,
            poni2=90.7 * 172e-6, rot1=0.01, rot2=-0.02, wavelength=1e-10)
FLAGS = N.DG_ERRORS | N.DG_AZIMUTHAL_STD


def _call(fn, plan, x, outs, stream):
    N.check(fn(plan.handle, C.c_void_p(x.data_ptr()), N.DG_U32, x.shape[0], FLAGS,
               *[C.c_void_p(o.data_ptr()) for o in outs],
               C.c_void_p(stream.cuda_stream) if stream is not None else None))


@pytest.mark.parametrize("variant", [7, 8, 10, 0])
@pytest.mark.parametrize("shape,bins", [((701, 899), 50), ((160, 200), 300)])  # cut tiles and whole ones
def test_capture_on_another_stream_than_the_warm_up(variant, shape, bins):
    import torch
    it = dg.Integrator.from_poni_dict(GEOM, method="pixel_split")
    plan = it.prepare_cuda1d(shape, bins)
    plan.gather_variant = variant
    L, n = N.lib(), 70
    gen = torch.Generator(device="cuda").manual_seed(1)

    def frames():
        return torch.randint(0, 2000, (n,) + shape, generator=gen, device="cuda", dtype=torch.int32)

    def outs():
        return [torch.full((n, bins), -1.0, dtype=torch.float64, device="cuda") for _ in range(3)]

    def plain(x, stream=None):
        o = outs()
        torch.cuda.synchronize()
        _call(L.dg_integrate_device, plan, x, o, stream)
        torch.cuda.synchronize()
        return o

    def same(a, b):
        return all(torch.equal(p.view(torch.int64), q.view(torch.int64)) for p, q in zip(a, b))

    x, y = frames(), frames()
    first = outs()
    torch.cuda.synchronize()
    _call(L.dg_integrate_device_noalloc, plan, x, first, None)  # warm-up
    want_x, want_y = plain(x), plain(y)
    assert same(first, want_x)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    still, got = x.clone(), outs()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        _call(L.dg_integrate_device_noalloc, plan, still, got, side)
    for src, want in ((x, want_x), (y, want_y), (x, want_x)):
        still.copy_(src)
        for o in got:
            o.fill_(-1.0)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert same(got, want)
    assert same(plain(y, other), want_y)  # a plain call on another stream goes on
    beside = outs()
    torch.cuda.synchronize()
    for _ in range(30):
        with torch.cuda.stream(side):
            graph.replay()
        _call(L.dg_integrate_device, plan, y, beside, other)
    torch.cuda.synchronize()
    assert same(got, want_x) and same(beside, want_y)
    del graph
    plan.close()
