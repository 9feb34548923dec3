"""Launch shape of claire_b200_reg_apply_noalloc's x1 pass.

On grids this small one CTA per column group and field is the faster shape
(64^3: 4.5 us, 6.5 with the three fields in one CTA), as in the allocating
entry point.  The launch is read from a trace, in a process of its own.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes, json, sys, torch
import claire_b200 as cb
from torch.profiler import profile, ProfilerActivity
n = int(sys.argv[1])
v = torch.randn((3, n, n, n), device="cuda")
out = torch.empty_like(v)
nx, beta = (ctypes.c_int * 3)(n, n, n), (ctypes.c_double * 2)(1e-3, 1e-4)
def call(name):
    f = getattr(cb.lib, name)
    assert f(ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(out.data_ptr()), nx, 4, beta, 1,
             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
names = ("claire_b200_reg_apply", "claire_b200_reg_apply_noalloc")
for name in names:
    call(name)
with profile(activities=[ProfilerActivity.CUDA]) as p:
    for name in names:
        call(name)
p.export_chrome_trace(sys.argv[2])
"""


@pytest.mark.parametrize("n", [16, 32, 48, 64])
def test_same_x1_grid_as_the_allocating_entry_point(cuda, tmp_path, n):
    trace = str(tmp_path / "trace.json")
    subprocess.run([sys.executable, "-c", SCRIPT, str(n), trace], cwd=ROOT, check=True, timeout=180)
    with open(trace) as f:
        grids = [e["args"]["grid"] for e in json.load(f)["traceEvents"]
                 if e.get("cat") == "kernel" and "k_pencil1" in e["name"]]
    assert len(grids) == 2
    assert grids[0] == grids[1]
