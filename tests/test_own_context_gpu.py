"""The library in a CUDA context of the caller's own (driver API) instead of the
device's primary one: device tree builds (whose shading arrays are uploaded by a
second thread), queries and a render, in a process of their own, equal to those
in the primary context, which is never made."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes as C, sys
import numpy as np
from bulbit_b200 import lib, scenes

own, out = sys.argv[1] == "own", sys.argv[2]
cu = C.CDLL("libcuda.so.1")
ctx = C.c_void_p()
if own:
    assert cu.cuInit(0) == 0 and cu.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0
scene = scenes.cornell_icosphere(levels=4, width=48, height=40, spp=4, max_bounces=6)
rays, _ = scenes.soup_rays(20_000, seed=3)
got = {}
for name, kw in (("sah", dict(device_sah=True)), ("split", dict(device_sah=True, split=1.0)),
                 ("linear", dict(device_build=True))):
    acc = lib.GpuAccel(scene, **kw)
    prim, t, u, v = acc.intersect(rays)
    got[name + "_hits"] = np.stack([prim.view(np.float32), t, u, v], 1).view(np.uint32)
    integ = lib.GpuPathIntegrator(acc, scene)
    got[name + "_film"] = integ.render().rgb_sum
    integ.close()
    acc.close()
now = C.c_void_p()
assert cu.cuCtxGetCurrent(C.byref(now)) == 0
assert not own or now.value == ctx.value, "the caller's context is no longer current"
flags, active = C.c_uint(), C.c_int()
assert cu.cuDevicePrimaryCtxGetState(0, C.byref(flags), C.byref(active)) == 0
assert active.value == (0 if own else 1), "work went to the device's primary context"
np.savez(out, **got)
if own:
    assert cu.cuCtxDestroy_v2(ctx) == 0
"""


def test_callers_own_context(tmp_path):
    res = {}
    for which in ("primary", "own"):
        out = str(tmp_path / f"{which}.npz")
        r = subprocess.run([sys.executable, "-c", CHILD, which, out], cwd=ROOT, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        res[which] = np.load(out)
    for k in res["primary"].files:
        assert np.array_equal(res["primary"][k], res["own"][k]), k
        assert res["own"][k].any()
