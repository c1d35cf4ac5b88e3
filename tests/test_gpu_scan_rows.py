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
