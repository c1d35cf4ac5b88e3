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
