"""One thread's stream capture and another thread's plans: creating a plan, growing
its scratch and destroying it leave a thread-local or relaxed capture intact, and a
destruction still waits for the plan's queued work."""
import ctypes as C
import threading

import pytest

import dioptrin_b200 as dg
from dioptrin_b200 import _native as N

pytestmark = pytest.mark.gpu

SHAPE, BINS = (160, 200), 300
GEOM = dict(pixel1=172e-6, pixel2=172e-6, distance=0.08, poni1=60.3 * 172e-6,
            poni2=75.7 * 172e-6, rot1=0.02, rot2=-0.01, wavelength=1e-10)


def _plan(variant):
    plan = dg.Integrator.from_poni_dict(GEOM, method="pixel_split").prepare_cuda1d(SHAPE, BINS)
    plan.gather_variant = variant
    return plan


def _frames(torch, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    return torch.randint(0, 2000, (n,) + SHAPE, generator=g, device="cuda", dtype=torch.int32)


def _call(fn, plan, x, out, stream=None):
    N.check(fn(plan.handle, C.c_void_p(x.data_ptr()), N.DG_U32, x.shape[0], 0,
               C.c_void_p(out.data_ptr()), None, None,
               C.c_void_p(stream.cuda_stream) if stream is not None else None))


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_other_threads_leave_a_capture_intact(mode):
    import torch
    L = N.lib()
    few, many = _frames(torch, 2), _frames(torch, 200)
    out, got = (torch.empty(200, BINS, dtype=torch.float64, device="cuda") for _ in range(2))
    plan, doomed = _plan(0), _plan(0)
    _call(L.dg_integrate_device, plan, many, out)  # sizes the scratch
    _call(L.dg_integrate_device, doomed, few, got)
    torch.cuda.synchronize()
    errors = []

    def others():
        try:
            _call(L.dg_integrate_device, doomed, many, got)  # grows: the old scratch is freed
            doomed.close()
            _plan(8).close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    side = torch.cuda.Stream()
    captured = torch.empty_like(out)
    graph = torch.cuda.CUDAGraph()
    _call(L.dg_integrate_device, plan, many, captured, side)  # so that no other stream's event is waited for
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side, capture_error_mode=mode):
        _call(L.dg_integrate_device, plan, many, captured, side)
        t = threading.Thread(target=others)
        t.start()
        t.join()
    assert not errors, errors
    captured.fill_(-1.0)
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, out) and torch.equal(got, out)
    del graph
    plan.close()
