"""The mesh convolution's passes at the sizes where they change form.

Meshes whose axes have two factors among 1..10, 12, 15 and 16 take the two-step passes
(csrc/fft.cuh): the narrow instance up to factors of 8, the wide one above, a plane's first
axis in one chunk or several (shared memory).  A length without such factors (a prime above
7, or a smooth one as 98, 125 or 162), or a plane beyond one CTA, takes the per-axis passes.  A 300-atom water box is evaluated on meshes of every
form, odd and prime lengths among them, against the FP64 oracle: the plain form at the
parity bar of test_gpu_parity (1e-8 relative per term, 1e-6 RMS gradient), the mixed form
at its own (test_gpu_precision_mixed) and bit for bit on repeated calls.
"""
import numpy as np
import pytest

from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import PRECISION_FP64, PRECISION_MIXED, small_water_box, water_params
from oracle import binding as ob

pytestmark = pytest.mark.gpu

MESHES = [
    (16, 16, 16), (15, 21, 28), (18, 27, 45),      # narrow and wide factors, odd lengths
    (5, 7, 64), (64, 14, 8),                       # a factor of one, unequal axes
    (64, 64, 64), (96, 80, 72), (120, 128, 10),    # one chunk, several chunks, factor 16
    (160, 160, 6),                                 # a plane beyond one CTA: per-axis passes
    (11, 20, 24), (20, 13, 16), (16, 18, 17),      # a general prime along each axis
    (64, 16, 11), (16, 64, 13), (16, 11, 64),      # per-axis passes of length 64, each kind
    (125, 12, 8), (10, 98, 12), (12, 10, 162),     # smooth lengths without two factors
]


@pytest.mark.parametrize("mesh", MESHES, ids=lambda m: "x".join(map(str, m)))
def test_convolution_forms(mesh):
    s, edge = small_water_box(300, seed=12)
    ref = None
    for precision in (PRECISION_FP64, PRECISION_MIXED):
        p = water_params(edge, pme_grid=mesh, precision=precision)
        ref = ref or ob.energy(s, p)
        with ForceFieldEnergy(s, p) as ffe:
            _, g = ffe.energy_and_gradient(s.xyz)      # direct launches
            _, g = ffe.energy_and_gradient(s.xyz)      # the captured graph
            terms, g = ffe.terms.copy(), g.copy()
            _, g2 = ffe.energy_and_gradient(s.xyz)
            terms2 = ffe.terms.copy()
        err = np.abs(terms - ref["terms"])
        rms = float(np.sqrt(np.mean((g - ref["grad"]) ** 2)))
        if precision == PRECISION_FP64:
            assert (err <= 1e-8 * np.maximum(np.abs(ref["terms"]), 1.0)).all(), err
            assert rms < 1e-6, rms
        else:
            assert err.max() < 1e-5 * abs(ref["terms"][9]), err
            assert rms < 1e-3, rms
            assert np.array_equal(terms, terms2) and np.array_equal(g, g2)
