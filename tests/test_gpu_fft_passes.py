"""The mesh passes as they are launched, from the activity trace.

A mesh that does not take the two-step passes goes through five passes, one axis each
(csrc/pme.cu, k_fft_axis).  The bars compare passes of one run with one another, medians over
its launches, so that neither the clock nor other work on the device decides them.  For the
two-step passes the shared memory of a plane's block shows in how many chunks it is taken.
"""
import json
import os
import re
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# In a process of its own: the activity trace stays out of the other tests.
TRACE = """
import json, sys, tempfile
import numpy as np, torch
from torch.profiler import ProfilerActivity, profile
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import small_water_box, water_params
mesh, precision = json.loads(sys.argv[1])
s, edge = small_water_box(300, seed=12)
with ForceFieldEnergy(s, water_params(edge, pme_grid=mesh, precision=precision)) as f:
    f.set_graph_mode(False)
    f.energy_and_gradient(s.xyz)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(3):
            f.energy_and_gradient(s.xyz)
        torch.cuda.synchronize()
with tempfile.NamedTemporaryFile(suffix=".json") as t:
    prof.export_chrome_trace(t.name)
    ev = [e for e in json.load(open(t.name))["traceEvents"] if e.get("cat") == "kernel"]
ev.sort(key=lambda e: e["ts"])
print(json.dumps([[e["name"], e["dur"], e["args"]["shared memory"]] for e in ev if "k_fft_" in e["name"]]))
"""


def _trace(mesh, precision):
    """(name, time in us, shared memory in bytes) of every transform launch of three evaluations."""
    env = dict(os.environ, PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", TRACE, json.dumps([mesh, precision])], env=env, cwd=ROOT, check=True,
                         capture_output=True, text=True, timeout=300).stdout
    return json.loads(out.strip().splitlines()[-1])


def _passes(mesh, precision):
    """Median time (us) of each of a convolution's five passes: x, y, z, y, x."""
    ev = _trace(mesh, precision)
    assert ev and len(ev) % 5 == 0
    fused = [bool(re.search(r"k_fft_axis<(true|1)", n)) for n, _, _ in ev]
    assert fused == [False, False, True, False, False] * (len(ev) // 5)
    return np.median(np.array([d for _, d, _ in ev]).reshape(-1, 5), axis=0)


def test_first_pass_keeps_its_loads_in_flight():
    """The first x pass reads the accumulation planes, clears them and writes the complex
    mesh: 96 bytes a point in FP64, cleared lines among them, where the last x pass moves 64
    with the same arithmetic.  Half as many again is 1.5; the bar is 2.  (With each load
    behind the store that clears the item before it, the ratio was 2.6 to 3.5.)"""
    x0, _, _, _, x1 = _passes((128, 128, 128), 0)
    assert x0 < 2.0 * x1, (x0, x1)


@pytest.mark.parametrize("precision", [0, 1])
def test_length_64_passes_without_run_time_divisions(precision):
    """A 48 x 64 x 77 mesh, 16 lines a block along x and y: the y pass (length 64, radix 4
    three times) has as many points and stages as the x pass (length 48, radices 4, 4 and 3),
    and its indices need no run-time division, half of the x pass: the bar is 0.65 of its
    time."""
    _, _, _, y, x = _passes((48, 64, 77), precision)
    assert y < 0.65 * x, (x, y)


@pytest.mark.parametrize("n,f1,f2,precision,chunks", [
    (32, 4, 8, 0, 1),        # the whole plane under 100 KB
    (64, 8, 8, 0, 4),        # the fewest that bring it there
    (80, 8, 10, 0, 9), (100, 10, 10, 0, 9), (128, 8, 16, 1, 9)])   # none of eight does
def test_chunks_of_a_plane(n, f1, f2, precision, chunks):
    """n lines of f1 runs of f2 values at odd strides, of each chunk and of the whole plane,
    and two twiddle tables: what fits beside a vdW block (17 KB) in an SM's 228 KB."""
    value = 8 if precision else 16
    stride = f1 * (f2 | 1) | 1
    want = ((-(-n // chunks) + n) * stride + 2 * n) * value
    assert want + 19 * 1024 <= 228 * 1024
    got = {sm for name, _, sm in _trace((n, n, 5), precision) if "k_fft_plane" in name}
    assert got == {want}, (got, want)
