"""Plans made after a device reset: the reset takes every kernel's raised
shared-memory limit with it, so the library has to raise them again.  In a
process of its own, which a reset leaves without a usable torch."""
from __future__ import annotations

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes
import sys

import numpy as np

lib = ctypes.CDLL(sys.argv[1])
lib.sht_last_error.restype = ctypes.c_char_p
driver = ctypes.CDLL("libcuda.so.1")
rng = np.random.default_rng(0)
P = ctypes.c_void_p


def ok(status):
    assert status == 0, lib.sht_last_error()


def round_trips():
    out = []
    # FP32 and split on the register FFTs, FP64 on the general ones: kernels
    # above the 48 KB that need no raised limit
    for precision in (1, 2, 0):
        plan = P()
        ok(lib.sht_plan_create(170, 256, 512, ctypes.c_double(6371220.0), precision, 0,
                               ctypes.byref(plan)))
        grid = np.ascontiguousarray(rng.standard_normal((6, 256, 512)),
                                    np.float64 if precision == 0 else np.float32)
        back = np.zeros_like(grid)
        for _ in range(2):
            ok(lib.sht_round_trip_host(plan, P(grid.ctypes.data), ctypes.c_int64(6),
                                       P(back.ctypes.data), ctypes.c_int64(0)))
        out.append(back)
    return out


first = round_trips()
assert driver.cuDevicePrimaryCtxReset_v2(0) == 0
rng = np.random.default_rng(0)
for a, b in zip(first, round_trips()):
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
"""


def test_plans_made_after_a_device_reset_launch():
    from b200sht import build

    done = subprocess.run([sys.executable, "-c", CHILD, str(build.LIB_PATH)], capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr


def test_a_capture_may_raise_the_limits():
    """A plan made after another was warm marks the limits as not raised; the
    warm plan's next launches raise them inside a stream capture."""
    import torch

    from b200sht import SphericalHarmonicTransform

    t = SphericalHarmonicTransform.create(169, nlat=256, nlon=512)
    grid = torch.randn(6, 256, 512, device="cuda")
    want = t.inverse(t.forward(grid))
    SphericalHarmonicTransform.create(21, nlat=33, nlon=66)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = t.inverse(t.forward(grid))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
