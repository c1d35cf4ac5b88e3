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


MODULES = """
import json, tempfile
import torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import small_water_box, water_params
torch.zeros(1, device="cuda")
s, edge = small_water_box(300, seed=12)
with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
    with ForceFieldEnergy(s, water_params(edge, pme_grid=(20, 20, 20))) as f:
        f.energy(s.xyz)
with tempfile.NamedTemporaryFile(suffix=".json") as t:
    prof.export_chrome_trace(t.name)
    ev = json.load(open(t.name))["traceEvents"]
name = {e["args"]["correlation"]: e["name"] for e in ev if e.get("cat") == "kernel"}
host = [(e["ts"], name[e["args"]["correlation"]], e["dur"]) for e in ev
        if e.get("cat") == "cuda_runtime" and e["args"].get("correlation") in name]
first = lambda k: next(d for _, n, d in sorted(host) if k in n)
print(json.dumps([first("k_rotate"), first("k_pack_mpole")]))
"""


def test_the_transforms_load_as_fast_as_the_pair_kernels():
    """A module is loaded by the first launch out of it: of pme.cu's the rotation (a 20^3 mesh
    needs no limit set before), of real.cu's the packing of the records.  The two modules
    hold 3.4 and 1.0 MB of code, read once from the library, the second 3 MB of line tables
    too, so that the first may take three times as long as the second, least of three
    processes; with 13 MB of line tables beside its code it took six times as long."""
    t = []
    for _ in range(3):
        out = subprocess.run([sys.executable, "-c", MODULES], env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT,
                             check=True, capture_output=True, text=True, timeout=300).stdout
        t.append(json.loads(out.strip().splitlines()[-1]))
    rotate, pack = (min(x) for x in zip(*t))
    assert rotate < 3.0 * pack, t
