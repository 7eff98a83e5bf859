"""The first step of a process: a kernel's first launch loads the module that
holds it.  The modules hold what a run uses together, uncompressed, so that a
program's first step waits a few milliseconds at most (with every kernel of a
precision in one compressed module: 4 ms in FP64, 12 in FP32).  The bounds are
twice what one kernel shape per module took (1.1 to 1.3 and 3.5 ms)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = r"""
import ctypes as C, sys, time
sys.path.insert(0, sys.argv[1])
from cuda.bindings import runtime as rt
from rapidsolid import _abi, configs, lib
f64 = sys.argv[2] == "f64"
p = configs.small(256, 256, i_tip_target=16, G=5e6, V=0.5)
ctx = lib.Context(p)
size = 256 * 256 * (8 if f64 else 4)
ptr = []
for _ in range(4):
    e, q = rt.cudaMalloc(size)
    assert int(e) == 0
    rt.cudaMemset(q, 0, size)
    ptr.append(q)
rt.cudaDeviceSynchronize()
prec = _abi.RS_F64 if f64 else _abi.RS_F32
cur, nxt = _abi.Fields(ptr[0], ptr[1], None, prec, 0), _abi.Fields(ptr[2], ptr[3], None, prec, 0)
a = _abi.StepArgs()
t0 = time.perf_counter()
lib.check(ctx.lib.rs_step(ctx._h, C.byref(cur), C.byref(nxt), C.byref(a), C.c_void_p(0)))
rt.cudaDeviceSynchronize()
print((time.perf_counter() - t0) * 1e3)
"""


@pytest.mark.parametrize("precision,ms", [("f64", 2.6), ("f32", 7.0)])
def test_first_step_of_a_process_loads_little(precision, ms):
    pkg = os.path.join(ROOT, "2d-rapid-solidification_b200")
    took = []
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", SCRIPT, pkg, precision], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        took.append(float(r.stdout.split()[-1]))
    assert min(took) <= ms, took
