"""What a process's first handle loads.

Setting a kernel's shared-memory limit loads the kernel, so a handle sets it for the passes
its mesh takes and only where they need more than every kernel has.  The calls are counted in
the activity trace of a fresh process.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

TRACE = """
import json, sys, tempfile
import torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import small_water_box, water_params
s, edge = small_water_box(300, seed=12)
out = []
for mesh, precision in json.loads(sys.argv[1]):
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
        f = ForceFieldEnergy(s, water_params(edge, pme_grid=mesh, precision=precision))
    f.close()
    with tempfile.NamedTemporaryFile(suffix=".json") as t:
        prof.export_chrome_trace(t.name)
        ev = [e["name"] for e in json.load(open(t.name))["traceEvents"] if e.get("cat") == "cuda_runtime"]
    assert "cudaMalloc" in ev
    out.append(ev.count("cudaFuncSetAttribute"))
print(json.dumps(out))
"""


def test_shared_memory_limits_are_set_where_they_are_needed():
    """Counts of the single-system and batch instances of each pass: none at 20^3; the two
    plane passes in mixed form at 64^3 (75 KB; the z pass stays below) and, the wide instances
    this time (60 = 6 x 10), at 60^3; none again at 56^3, which needs no more than 64^3; the
    three per-axis passes of 128^3 in FP64 (64 KB), and none again for 125 x 120 x 128."""
    cases = [([20, 20, 20], 0), ([64, 64, 64], 1), ([60, 60, 60], 1), ([56, 56, 56], 1), ([128, 128, 128], 0),
             ([125, 120, 128], 0)]
    out = subprocess.run([sys.executable, "-c", TRACE, json.dumps(cases)], env=dict(os.environ, PYTHONPATH=ROOT),
                         cwd=ROOT, check=True, capture_output=True, text=True, timeout=300).stdout
    assert json.loads(out.strip().splitlines()[-1]) == [0, 4, 4, 0, 6, 0]
