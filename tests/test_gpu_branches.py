"""When a captured evaluation starts its vdW branch, from the activity trace.

vdW runs at one block a multiprocessor beside the solver: after the real-space field, where it
ends before the solver does, and at once with more atoms (csrc/handle.cu, vdw_late_atoms).
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# In a process of its own: the activity trace stays out of the other tests.
TRACE = """
import json, sys, tempfile
import torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import water_box, water_params
n_side, mesh, precision = json.loads(sys.argv[1])
edge = n_side * 3.104
s = water_box(n_side, edge, seed=3)
with ForceFieldEnergy(s, water_params(edge, pme_grid=(mesh,) * 3, precision=precision)) as f:
    for _ in range(3):
        f.energy_and_gradient(s.xyz)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        f.energy_and_gradient(s.xyz)
        torch.cuda.synchronize()
with tempfile.NamedTemporaryFile(suffix=".json") as t:
    prof.export_chrome_trace(t.name)
    ev = [e for e in json.load(open(t.name))["traceEvents"] if e.get("cat") == "kernel"]
vdw = [e for e in ev if "k_vdw<" in e["name"]]
field = [e for e in ev if "k_realspace_field" in e["name"]]
assert len(vdw) == len(field) == 1
print(json.dumps([vdw[0]["ts"] - field[0]["ts"], field[0]["dur"]]))
"""


@pytest.mark.parametrize("n_side,mesh,precision,late", [(20, 64, 0, True), (20, 64, 1, True), (28, 90, 0, False),
                                                        (30, 96, 1, True), (37, 120, 1, False)])
def test_vdw_branch_starts_after_the_field_up_to_its_size(n_side, mesh, precision, late):
    out = subprocess.run([sys.executable, "-c", TRACE, json.dumps([n_side, mesh, precision])],
                         env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT, check=True, capture_output=True, text=True,
                         timeout=300).stdout
    start, field = json.loads(out.strip().splitlines()[-1])   # from the field's start, and its time
    assert (start > 0.5 * field) == late, (start, field)


OVERLAP = """
import json, sys, tempfile, time
import torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import water_box, water_params
edge = 40 * 3.104
s = water_box(40, edge, seed=3)
x = torch.tensor(s.xyz, device="cuda")
g = torch.empty_like(x)
with ForceFieldEnergy(s, water_params(edge, pme_grid=(128, 128, 128), precision=0)) as f:
    t = []
    for _ in range(10):
        a = time.perf_counter()
        f.energy_device(x.data_ptr(), g.data_ptr())
        t.append(time.perf_counter() - a)
    f.set_graph_mode(False)
    f.energy_device(x.data_ptr(), g.data_ptr())
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        f.energy_device(x.data_ptr(), g.data_ptr())
with tempfile.NamedTemporaryFile(suffix=".json") as tmp:
    prof.export_chrome_trace(tmp.name)
    ev = [e for e in json.load(open(tmp.name))["traceEvents"] if e.get("cat") == "kernel"]
print(json.dumps([1e6 * sorted(t)[4], sum(e["dur"] for e in ev)]))
"""


def test_branches_overlap_on_a_large_per_axis_mesh():
    """192,000 atoms on a 128^3 mesh in FP64, whose passes (64 KB a block) run beside vdW only
    where the shared-memory split of its blocks leaves them room: vdW (a fifteenth of the
    kernels' time alone) and the spreads, transforms and pair fields of each iteration (half)
    overlap, for at least an eighth of the total."""
    out = subprocess.run([sys.executable, "-c", OVERLAP], env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT, check=True,
                         capture_output=True, text=True, timeout=300).stdout
    captured, kernels = json.loads(out.strip().splitlines()[-1])
    assert captured < 0.87 * kernels, (captured, kernels)
