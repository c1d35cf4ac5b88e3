"""Row scans of multi-image lists against those of minimum-image lists, from the activity trace.

The real-space field queues what a row's cheap test passes and works on full warps
(csrc/ffx_internal.cuh).  A 3,000-atom box is evaluated with its minimum-image lists and with
every image listed: the same pairs lie inside the cutoff.
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
from forcefieldx_b200.system import small_water_box, water_params
s, edge = small_water_box(3000, seed=4)
out = []
for images in (False, True):
    with ForceFieldEnergy(s, water_params(edge, pme_grid=(32, 32, 32), precision=int(sys.argv[1]))) as f:
        f.set_graph_mode(False)
        f.set_image_mode(images)
        f.energy_and_gradient(s.xyz)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(7):
                f.energy_and_gradient(s.xyz)
            torch.cuda.synchronize()
    with tempfile.NamedTemporaryFile(suffix=".json") as t:
        prof.export_chrome_trace(t.name)
        ev = json.load(open(t.name))["traceEvents"]
    d = sorted(e["dur"] for e in ev if e.get("cat") == "kernel" and "k_realspace_field" in e["name"])
    assert len(d) == 7
    out.append(d[3])
print(json.dumps(out))
"""


@pytest.mark.parametrize("precision", [0, 1])
def test_field_of_a_multi_image_list_works_on_full_warps(precision):
    """The multi-image list scans the 11 A rows, the minimum-image one the near rows of
    9.5 A: 1.55 times as many entries in the scan, as many in the pair arithmetic, and the
    same tests.  The bar is 1.6 for the whole kernel; pair arithmetic on every entry listed
    would take four times as many pairs."""
    out = subprocess.run([sys.executable, "-c", TRACE, str(precision)], env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT,
                         check=True, capture_output=True, text=True, timeout=300).stdout
    plain, images = json.loads(out.strip().splitlines()[-1])
    assert images < 1.6 * plain, (plain, images)


BATCH = """
import json, sys, tempfile
import torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.batch import BatchEnergy
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import WATER_24K, small_water_box, water_box, water_params
precision = int(sys.argv[1])
def vdw(call):
    call(); call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(5):
            call()
        torch.cuda.synchronize()
    with tempfile.NamedTemporaryFile(suffix=".json") as t:
        prof.export_chrome_trace(t.name)
        ev = json.load(open(t.name))["traceEvents"]
    d = sorted(e["dur"] for e in ev if e.get("cat") == "kernel" and "k_vdw<" in e["name"])
    assert len(d) == 5
    return d[2]
s = water_box(WATER_24K["n_side"], WATER_24K["edge"])
with ForceFieldEnergy(s, water_params(WATER_24K["edge"], pme_grid=WATER_24K["grid"], precision=precision)) as f:
    f.set_graph_mode(False)
    single = vdw(lambda: f.energy_and_gradient(s.xyz)) / s.n_atoms
w = []
for k in range(32):
    s, edge = small_water_box(3000, seed=k)
    w.append((s, water_params(edge, pme_grid=(32, 32, 32), precision=precision)))
with BatchEnergy([a for a, _ in w], [b for _, b in w]) as b:
    b.set_groups(1)
    batch = vdw(lambda: b.energy_and_gradient([a.xyz for a, _ in w])) / 96000
print(json.dumps([single, batch]))
"""


@pytest.mark.parametrize("precision", [0, 1])
def test_vdw_of_a_batch_costs_what_a_single_box_does(precision):
    """The same pairs per atom in 32 boxes of 3,000 atoms in one launch as in one box of
    24,000; the batch has four times the atoms, so that its last wave weighs less, and its
    instance may hold fewer resident warps: 1.4 times the single box's time per atom."""
    out = subprocess.run([sys.executable, "-c", BATCH, str(precision)], env=dict(os.environ, PYTHONPATH=ROOT), cwd=ROOT,
                         check=True, capture_output=True, text=True, timeout=300).stdout
    single, batch = json.loads(out.strip().splitlines()[-1])
    assert batch < 1.4 * single, (single, batch)
