"""Plans after cudaDeviceReset: memory, streams and pools of the library end with
the context, and a plan made afterwards works (in a process of its own, which
destroys its plans before it resets)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
import numpy as np
import dioptrin_b200 as dg
import glob, os, importlib.util
root = os.path.dirname(importlib.util.find_spec("nvidia.cuda_runtime").submodule_search_locations[0])
rt = ctypes.CDLL(glob.glob(os.path.join(root, "cuda_runtime", "lib", "libcudart.so*"))[0])
geom = dict(pixel1=172e-6, pixel2=172e-6, distance=0.08, poni1=0.01, poni2=0.012, wavelength=1e-10)
frames = np.random.default_rng(1).integers(0, 900, (40, 160, 200)).astype(np.uint32)
want = None
for turn in range(3):
    plan = dg.Integrator.from_poni_dict(geom, method="pixel_split").prepare_cuda1d((160, 200), 300)
    for variant in (0, 8, 10):
        plan.gather_variant = variant
        got = plan.integrate_stack(frames, True, True)
    if want is None:
        want = got
    assert all(a.tobytes() == b.tobytes() for a, b in zip(got, want))
    plan.close()
    if turn < 2:
        assert rt.cudaDeviceReset() == 0
print("three plans, two resets")
"""


def test_plans_after_a_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=120,
                       cwd=root)
    assert r.returncode == 0 and "three plans, two resets" in r.stdout, r.stdout + r.stderr
