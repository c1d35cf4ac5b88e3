"""Row scans where the fixed-point test and the one-addition wrap change branch.

The vdW and real-space field kernels first test a row's entries on 32-bit fixed-point
fractions (csrc/ffx_internal.cuh: fixed_r2) and take the exact minimum image of what
passes, wrapping by one addition below 3/2 of an edge and by the general rounding beyond.
Molecules of a water box are carried whole lattice vectors away (none, a neighbouring cell,
tens of cells), in an orthorhombic and a triclinic cell, and the interaction counts must
equal the oracle's exactly; energies and gradients meet the FP64 parity bar (1e-8 relative
per term, 1e-6 RMS) or the mixed form's (1e-5 of the total, 1e-3 RMS).

In a triclinic cell whose half width the list reaches, a pair half a cell apart has two images
at different distances, and the fixed-point fractions may wrap to the other one than the exact
test takes: the builder then tests every candidate exactly (csrc/nlist.cu).
"""
import numpy as np
import pytest

from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import PRECISION_FP64, PRECISION_MIXED, water_box, water_params
from oracle import binding as ob

pytestmark = pytest.mark.gpu

EDGE = 23.3


def _lattice(angles, edge=EDGE):
    """Rows a, b, c of the cell with these edges and angles (degrees)."""
    al, be, ga = np.radians(angles)
    bx, by = np.cos(ga), np.sin(ga)
    cx = np.cos(be)
    cy = (np.cos(al) - np.cos(be) * np.cos(ga)) / np.sin(ga)
    return edge * np.array([[1, 0, 0], [bx, by, 0], [cx, cy, np.sqrt(1 - cx * cx - cy * cy)]])


@pytest.mark.parametrize("reach", [0, 1, 40])
@pytest.mark.parametrize("angles", [(90.0, 90.0, 90.0), (82.0, 97.0, 88.0)], ids=["ortho", "triclinic"])
def test_scan_over_lattice_translations(angles, reach):
    s = water_box(7, EDGE, seed=8)
    rng = np.random.default_rng(5 + reach)
    shift = rng.integers(-reach, reach + 1, size=(s.n_atoms // 3, 3))
    x = s.xyz + np.repeat(shift @ _lattice(angles), 3, axis=0)
    for precision in (PRECISION_FP64, PRECISION_MIXED):
        p = water_params(EDGE, pme_grid=(24, 24, 24), precision=precision, angles=angles)
        ref = ob.energy(s, p, xyz=x)
        assert ref["status"] == 0
        with ForceFieldEnergy(s, p) as ffe:
            for _ in range(2):                     # direct launches, then the captured graph
                _, g = ffe.energy_and_gradient(x)
            terms, counts = ffe.terms.copy(), ffe.counts.copy()
        assert counts[0] == ref["counts"][0] and counts[1] == ref["counts"][1]
        err = np.abs(terms - ref["terms"])
        rms = float(np.sqrt(np.mean((g - ref["grad"]) ** 2)))
        if precision == PRECISION_FP64:
            assert (err <= 1e-8 * np.maximum(np.abs(ref["terms"]), 1.0)).all(), err
            assert rms < 1e-6, rms
        else:
            assert err.max() < 1e-5 * abs(ref["terms"][9]), err
            assert rms < 1e-3, rms


@pytest.mark.parametrize("precision", [PRECISION_FP64, PRECISION_MIXED])
def test_list_of_pairs_half_an_oblique_cell_apart(precision):
    """216 waters with their oxygens on a 6 x 6 x 6 grid of the cell, so that many oxygen
    pairs differ by half a lattice vector to rounding: 21 A edges, half width 10.3 A, an 11 A
    list of 9 A cutoffs.  The pair set must be the oracle's."""
    edge, angles = 21.0, (82.0, 97.0, 88.0)
    s = water_box(6, edge, seed=9, jitter=0.0)
    o = np.repeat(s.xyz[::3], 3, axis=0)
    s.xyz = s.xyz - o + (o / edge) @ _lattice(angles, edge)
    p = water_params(edge, pme_grid=(24, 24, 24), precision=precision, angles=angles)
    want = {(int(min(r)), int(max(r))) for r in ob.neighbor_pairs(s, p)}
    ref = ob.energy(s, p)
    assert ref["status"] == 0
    with ForceFieldEnergy(s, p) as ffe:
        for _ in range(2):                     # direct launches, then the captured graph
            _, g = ffe.energy_and_gradient(s.xyz)
        rows, terms, counts = ffe.neighbor_pairs(), ffe.terms.copy(), ffe.counts.copy()
    got = {(int(min(r)), int(max(r))) for r in rows}
    assert len(got) == len(rows) and got == want
    assert counts[0] == ref["counts"][0] and counts[1] == ref["counts"][1]
    err = np.abs(terms - ref["terms"])
    rms = float(np.sqrt(np.mean((g - ref["grad"]) ** 2)))
    if precision == PRECISION_FP64:
        assert (err <= 1e-8 * np.maximum(np.abs(ref["terms"]), 1.0)).all(), err
        assert rms < 1e-6, rms
    else:
        assert err.max() < 1e-5 * abs(ref["terms"][9]), err
        assert rms < 1e-3, rms
