"""Work that programs have this library do, through its public entry points.

Every system is a periodic box of rigid AMOEBA waters on a seeded, jittered lattice with
random orientations at 1.0 g/cm^3, with the cutoffs of the water configurations (9 A vdW,
7 A real space, order 5, PCG to 1e-6 D).  A case is one of these kinds:

  gradient  ForceFieldEnergy.energy_and_gradient: host coordinates in, host gradient out,
            the call of an optimizer or of a host-side integrator
  energy    ForceFieldEnergy.energy: a Monte Carlo or barostat trial, no gradient
  md        ForceFieldEnergy.md_run: constant-energy dynamics of rigid waters on the device
  lambda    energy_and_gradient + get_dEdL of an alchemical window (softcore vdW and
            electrostatics of a few soft molecules)
  fit       energy_and_gradient + param_gradients: one step of parameter fitting
  batch     BatchEnergy.energy_and_gradient: many small systems of uneven size in one call
"""
import math

import numpy as np
import torch

from forcefieldx_b200.batch import BatchEnergy, pme_grid_for
from forcefieldx_b200.energy import ForceFieldEnergy
from forcefieldx_b200.system import (PRECISION_FP64, PRECISION_MIXED, Alchemy, tile_system, water_box,
                                     water_params)

VOLUME = 62.08 ** 3 / 8000      # A^3 per water molecule
SPACING = 0.97                  # A per PME mesh point: 64 over 62.08 A, 20 over 18.643 A
ROH, THETA = 0.9572, math.radians(104.52)
RHH = 2.0 * ROH * math.sin(THETA / 2.0)
MASS_O, MASS_H = 15.999, 1.008
KCAL = 418.4                    # kcal/mol in amu A^2 / ps^2
PCG_STEPS = 8                   # solver iterations of a water box at 1e-6 D, for work()


def listed():
    return [
        # The smallest box whose cutoffs fit: launches and latency decide.
        case("gradient-648-fp64", "gradient", "fp64", 216),
        # A small solvated molecule's box, uneven edges and an odd mesh.
        case("gradient-2997-mixed", "gradient", "mixed", 999, ry=1.13, rz=0.91),
        # A small protein's box (ubiquitin with its water is 9,737 atoms), uneven edges.
        case("gradient-9738-fp64", "gradient", "fp64", 3246, ry=0.93, rz=1.21),
        # The ordinary box, in both forms.
        case("gradient-24000-fp64", "gradient", "fp64", 8000),
        case("gradient-24000-mixed", "gradient", "mixed", 8000),
        # Trial moves of a barostat: energies alone.
        case("energy-9738-mixed", "energy", "mixed", 3246, ry=1.05, rz=0.88),
        # The largest: a membrane-sized box.
        case("gradient-81000-mixed", "gradient", "mixed", 27000),
        # Dynamics at 2 fs.
        case("md-24000-fp64", "md", "fp64", 8000, steps=8),
        # One alchemical window, ten soft waters.
        case("lambda-24000-fp64", "lambda", "fp64", 8000, lam=0.5, soft=10),
        # One step of a fit of multipoles and polarizabilities.
        case("fit-9738-fp64", "fit", "fp64", 3246, ry=1.05, rz=1.1),
        # Conformers or windows of small systems, evaluated together.
        case("batch-96-mixed", "batch", "mixed", 1000, systems=96),
    ]


def case(name, kind, precision, waters, ry=1.0, rz=1.0, steps=0, lam=1.0, soft=0, systems=0):
    c = {"kind": kind, "precision": precision, "waters": waters, "ry": ry, "rz": rz, "steps": steps, "lam": lam,
         "soft": soft, "systems": systems}
    return dict(c, name=name) if name else c


def draw(rng):
    kind = rng.choice(["gradient", "gradient", "gradient", "energy", "md", "lambda", "fit", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    ry, rz = round(rng.uniform(0.9, 1.25), 3), round(rng.uniform(0.9, 1.25), 3)
    if kind == "batch":
        return case(None, kind, precision, size(400, 1000), systems=rng.randint(12, 64))
    if kind == "md":
        return case(None, kind, "fp64", size(400, 8000), ry, rz, steps=rng.randint(2, 8))
    if kind == "lambda":
        return case(None, kind, "fp64", size(400, 8000), ry, rz, lam=round(rng.uniform(0.05, 0.7), 3),
                    soft=rng.randint(1, 12))
    if kind == "fit":
        return case(None, kind, "fp64", size(400, 8000), ry, rz)
    return case(None, kind, precision, size(400, 24000), ry, rz)


# ------------------------------------------------------------------------------------
def edges_of(c):
    """Box edges; 216 waters with ry = rz = 1 is the 18.643 A cube."""
    a = (c["waters"] * VOLUME / (c["ry"] * c["rz"])) ** (1.0 / 3.0)
    return a, a * c["ry"], a * c["rz"]


def water_lattice(waters, edges, rng, jitter=0.15):
    """[3 * waters, 3] coordinates: sites of a lattice that fits the box, drawn without
    replacement, each molecule turned at random."""
    edges = np.asarray(edges)
    k = np.maximum(1, np.round(edges / (edges.prod() / waters) ** (1.0 / 3.0))).astype(int)
    while k.prod() < waters:
        k[np.argmax(edges / k)] += 1
    sites = np.sort(rng.choice(k.prod(), size=waters, replace=False))
    grid = np.stack(np.unravel_index(sites, k), axis=1)
    origin = (grid + 0.5) * (edges / k) - 0.5 * edges + rng.uniform(-jitter, jitter, size=(waters, 3))
    q = rng.normal(size=(waters, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1)[:, None]).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                    2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                    2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], axis=1).reshape(-1, 3, 3)
    s, t = ROH * math.sin(THETA / 2), ROH * math.cos(THETA / 2)
    local = np.array([[0.0, 0.0, 0.0], [s, 0.0, t], [-s, 0.0, t]])
    return (origin[:, None, :] + np.einsum("wij,aj->wai", rot, local)).reshape(-1, 3)


def systems_of(c, seed):
    """[(system, params)]: one, or a batch's."""
    rng = np.random.default_rng(seed)
    precision = PRECISION_MIXED if c["precision"] == "mixed" else PRECISION_FP64
    one = water_box(1, 10.0, seed=1)
    out = []
    # A batch's sizes belong to the case: 96 atoms up to its largest, uniform, in any order.
    sizes = np.random.default_rng([c["systems"], c["waters"]]).integers(32, c["waters"] + 1, size=max(1, c["systems"]))
    for waters in sizes.tolist():
        if c["kind"] == "batch":
            edges = ((waters * 29.915) ** (1.0 / 3.0),) * 3
            mesh = (pme_grid_for(edges[0], 1.2),) * 3
            xyz = water_lattice(waters, edges, rng, jitter=0.1)
        else:
            waters, edges = c["waters"], edges_of(c)
            mesh = tuple(pme_grid_for(e, SPACING) for e in edges)
            xyz = water_lattice(waters, edges, rng)
        out.append((tile_system(one, xyz, waters),
                    water_params(edges[0], box=edges, pme_grid=mesh, precision=precision)))
    return out


def soft_atoms(c, seed):
    soft = np.zeros(3 * c["waters"], dtype=np.int32)
    for w in np.random.default_rng(seed + 1).choice(c["waters"], c["soft"], replace=False):
        soft[3 * w:3 * w + 3] = 1
    return soft


def masses(n):
    return np.where(np.arange(n) % 3 == 0, MASS_O, MASS_H)


def velocities(xyz, seed):
    """300 K, with no motion along the rigid sides."""
    m = masses(len(xyz))
    v = np.random.default_rng(seed + 2).normal(size=xyz.shape) * np.sqrt(0.0019872041 * 300.0 * KCAL / m)[:, None]
    return rattle(xyz, v)


def prepare(case, seed):
    work = systems_of(case, seed)
    s, p = work[0]
    if case["kind"] == "batch":
        return {"case": case, "handle": BatchEnergy([w[0] for w in work], [w[1] for w in work]),
                "xyz": [w[0].xyz for w in work]}
    handle = ForceFieldEnergy(s, p)
    state = {"case": case, "handle": handle, "xyz": s.xyz, "gradient": np.zeros_like(s.xyz)}
    if case["kind"] == "md":
        handle.md_setup(masses(s.n_atoms), np.arange(s.n_atoms).reshape(-1, 3), ROH, RHH)
        state["velocities"] = velocities(s.xyz, seed)
    if case["kind"] == "lambda":
        handle.set_alchemy(Alchemy(soft=soft_atoms(case, seed), molecule=np.arange(s.n_atoms) // 3, elec=True))
        handle.set_lambda(case["lam"])
    return state


def run(state):
    """The energy terms (the total among them) and what else the call returns."""
    kind, h = state["case"]["kind"], state["handle"]
    if kind == "batch":
        _, g = h.energy_and_gradient(state["xyz"])
        return {"terms": h.terms.copy(), "gradient": np.concatenate(g)}
    if kind == "md":
        x, v, ep, ek = h.md_run(state["xyz"], state["velocities"], 0.002, state["case"]["steps"])
        return {"xyz": x, "velocities": v, "epot": ep, "ekin": ek}
    if kind == "energy":
        h.energy(state["xyz"])
        return {"terms": h.terms.copy()}
    h.energy_and_gradient(state["xyz"], state["gradient"])
    out = {"terms": h.terms.copy(), "gradient": state["gradient"].copy()}
    if kind == "lambda":
        d1, d2, dx = h.get_dEdL()
        out.update(dEdL=np.array([d1, d2]), dEdXdL=dx)
    if kind == "fit":
        out["dEdM"], out["dEdalpha"] = h.param_gradients()
    return out


def work(case):
    """Bytes: coordinates and parameters read once, results written once.  Operations: each
    vdW pair and each real-space pair once per pass over it (110 for a dipole field, 900 for
    the energy), the mesh's spreads, interpolations and transforms."""
    atoms, points, vdw, real = 0.0, 0.0, 0.0, 0.0
    n = 3.0 * case["waters"]
    sizes = [n]
    if case["kind"] == "batch":
        sizes = [96 + (n - 96) * (j + 0.5) / case["systems"] for j in range(case["systems"])]
    for m in sizes:
        atoms += m
        points += m / 3.0 * VOLUME / SPACING ** 3
        per = 4.0 / 3.0 * math.pi * 3.0 / VOLUME * 0.5 * m
        vdw += per * 9.0 ** 3
        real += per * 7.0 ** 3
    wide = 4.0 if case["precision"] == "mixed" else 8.0
    solves = 2 if case["kind"] == "lambda" else 1
    mesh = 2 * 125 * 8 * atoms + 10.0 * points * math.log2(max(points, 2.0))
    flops = 70 * vdw + (900 + 110) * real + solves * PCG_STEPS * (2 * 110 * real + mesh) + 2 * mesh
    per_atom = 24 + 8 * 10 + 8 * 4 + 4 * 6 + (0 if case["kind"] == "energy" else 24) + wide * 6
    if case["kind"] == "lambda":
        per_atom += 24
    if case["kind"] == "fit":
        per_atom += 88
        flops += 600 * real
    passes = 1
    if case["kind"] == "md":
        passes = case["steps"] + 1
    return {"bytes": passes * per_atom * atoms, "flops": passes * flops}


# ------------------------------------------------------------------------------------
# The same results in 64 bits with torch: every pair by distance, the induced dipoles solved
# to 1e-13, gradients by automatic differentiation.
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def t64(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)


def pairs_within(xyz, edges, cutoff):
    """(i, k, shift, primary) of every image pair x_k + shift - x_i within the cutoff, each
    once; primary: the minimum image."""
    n, edges = len(xyz), torch.as_tensor(edges, device=DEV, dtype=torch.float64)
    reach = [int(math.floor(cutoff / float(e) + 0.5)) for e in edges]
    I, K, S, P = [], [], [], []
    rows = max(1, int(3e7) // n)
    for lo in range(0, n, rows):
        d = xyz[None, :, :] - xyz[lo:lo + rows, None, :]
        base = -torch.round(d / edges)
        at = torch.arange(lo, min(n, lo + rows), device=DEV)[:, None]
        upper = torch.arange(n, device=DEV)[None, :] > at
        same = torch.arange(n, device=DEV)[None, :] == at
        d = d + base * edges
        for mx in range(-reach[0], reach[0] + 1):
            for my in range(-reach[1], reach[1] + 1):
                for mz in range(-reach[2], reach[2] + 1):
                    m = torch.tensor([mx, my, mz], device=DEV, dtype=torch.float64)
                    keep = upper | same if (mx, my, mz) > (0, 0, 0) else upper
                    i, k = torch.nonzero(keep & (((d + m * edges) ** 2).sum(-1) <= cutoff * cutoff), as_tuple=True)
                    I.append(i + lo)
                    K.append(k)
                    S.append((base[i, k] + m) * edges)
                    P.append(torch.full_like(i, int((mx, my, mz) == (0, 0, 0)), dtype=torch.bool))
        del d, base
    return torch.cat(I), torch.cat(K), torch.cat(S), torch.cat(P)


def vdw_energy(x, inputs, lam):
    """Buffered 14-7 with the multiplicative taper; a pair of one soft and one hard atom is
    softened."""
    s, p = inputs["system"], inputs["params"]
    i, k, shift, primary = inputs["vdw_pairs"]
    f = t64(s.red_factor)[:, None]
    parent = torch.as_tensor(s.red_parent, device=DEV).long()
    r = torch.where(f > 0, f * (x - x[parent]) + x[parent], x)
    apart = ~(primary & (i // 3 == k // 3))
    i, k, shift = i[apart], k[apart], shift[apart]
    ty = torch.as_tensor(s.vdw_type, device=DEV).long()
    dist = ((r[k] + shift - r[i]) ** 2).sum(-1).sqrt()
    inside = dist <= p.vdw_cutoff
    i, k, dist = i[inside], k[inside], dist[inside]
    eps, inv = t64(s.vdw_eps)[ty[i], ty[k]], t64(s.vdw_inv_rmin)[ty[i], ty[k]]
    rho = dist * inv
    one = torch.ones_like(rho)
    soft = torch.as_tensor(inputs["soft"], device=DEV).bool()
    mixed = soft[i] != soft[k]
    a = torch.where(mixed, 0.25 * (1 - lam) ** 2 * one, 0.0)
    scale = torch.where(mixed, lam ** 3 * one, 1.0)
    e = scale * eps * 1.07 ** 7 / (a + (rho + 0.07) ** 7) * (1.12 / (a + rho ** 7 + 0.12) - 2.0)
    cut = p.vdw_taper * p.vdw_cutoff
    t = ((dist - cut) / (p.vdw_cutoff - cut)).clamp(min=0.0)
    return (e * (1.0 - 10.0 * t ** 3 + 15.0 * t ** 4 - 6.0 * t ** 5)).sum()


def global_multipoles(x, local):
    """Charges, dipoles and quadrupoles in the laboratory frame: the bisector frame of an
    oxygen, z-then-x of a hydrogen."""
    w = x.reshape(-1, 3, 3)
    unit = lambda v: v / (v * v).sum(-1, keepdim=True).sqrt()  # noqa: E731
    frames = []
    for o, a, b, bisector in ((0, 1, 2, True), (1, 0, 2, False), (2, 0, 1, False)):
        z, q = unit(w[:, a] - w[:, o]), w[:, b] - w[:, o]
        if bisector:
            q = unit(q)
            z = unit(z + q)
        q = unit(q - (q * z).sum(-1, keepdim=True) * z)
        frames.append(torch.stack([q, torch.cross(z, q, dim=-1), z], dim=-1))
    rot = torch.stack(frames, dim=1).reshape(-1, 3, 3)
    quad = local[:, [4, 7, 8, 7, 5, 9, 8, 9, 6]].reshape(-1, 3, 3)
    return local[:, 0], (rot @ local[:, 1:4, None])[..., 0], rot @ quad @ rot.transpose(1, 2)


def bn_factors(r, alpha, top):
    inv2 = 1.0 / (r * r)
    bn = [(torch.erfc(alpha * r) if alpha > 0 else torch.ones_like(r)) / r]
    e = torch.exp(-(alpha * r) ** 2) / (math.sqrt(math.pi) * alpha) if alpha > 0 else 0.0
    rr = [1.0 / r]
    for j in range(1, top):
        e = e * 2 * alpha * alpha
        bn.append(((2 * j - 1) * bn[-1] + e) * inv2)
        rr.append((2 * j - 1) * rr[-1] * inv2)
    return bn, rr


def thole_factors(r, s, i, k):
    pd, th = t64(s.pdamp), t64(s.thole)
    damp = -torch.minimum(th[i], th[k]) * (r / (pd[i] * pd[k])) ** 3
    e = torch.exp(damp)
    return 1 - e, 1 - e * (1 - damp), 1 - e * (1 - damp + 0.6 * damp * damp)


def dot(a, b):
    return (a * b).sum(-1)


def permanent_real(x, mult, pairs, alpha, soften=None):
    """Sum over pairs of the screened multipole energy; soften: (soft mask, added r^2, scale)."""
    i, k, shift, primary = pairs
    q, d, Q = mult
    Q = Q / 3.0
    v = x[k] + shift - x[i]
    r2, scale = dot(v, v), 1.0
    if soften is not None:
        r2 = r2 + torch.where(soften[0], soften[1], torch.zeros_like(r2))
        scale = torch.where(soften[0], soften[2], torch.ones_like(r2))
    bn, rr = bn_factors(r2.sqrt(), alpha, 5)
    drop = (primary & (i // 3 == k // 3)).double()
    b = [u - drop * w for u, w in zip(bn, rr)]
    qi, qk = (Q[i] @ v[..., None])[..., 0], (Q[k] @ v[..., None])[..., 0]
    di, dk, ci, ck = d[i], d[k], q[i], q[k]
    s3, s4, s5, s6 = dot(di, v), dot(dk, v), dot(qi, v), dot(qk, v)
    e = ci * ck * b[0] + (ck * s3 - ci * s4 + dot(di, dk)) * b[1]
    e = e + (ci * s6 + ck * s5 - s3 * s4 + 2 * (dot(qi, dk) - dot(qk, di)) + 2 * (Q[i] * Q[k]).sum((-1, -2))) * b[2]
    e = e + (s3 * s6 - s4 * s5 - 4 * dot(qi, qk)) * b[3] + s5 * s6 * b[4]
    return (scale * e).sum()


def field_dot(x, mult, u, s, pairs, alpha):
    """Sum over atoms of u . (masked, damped real-space field of the multipoles)."""
    i, k, shift, primary = pairs
    q, d, Q = mult
    Q = Q / 3.0
    v = x[k] + shift - x[i]
    r = dot(v, v).sqrt()
    bn, rr = bn_factors(r, alpha, 4)
    keep = (~(primary & (i // 3 == k // 3))).double()
    f = [bn[j + 1] - (1 - keep * t) * rr[j + 1] for j, t in enumerate(thole_factors(r, s, i, k))]
    qi, qk = 2 * (Q[i] @ v[..., None])[..., 0], 2 * (Q[k] @ v[..., None])[..., 0]
    a = f[0] * q[i] + f[1] * dot(d[i], v) + f[2] * dot(qi, v) * 0.5
    at_k = a[:, None] * v - f[0][:, None] * d[i] - f[1][:, None] * qi
    a = f[0] * q[k] - f[1] * dot(d[k], v) + f[2] * dot(qk, v) * 0.5
    at_i = -a[:, None] * v - f[0][:, None] * d[k] + f[1][:, None] * qk
    return dot(at_k, u[k]).sum() + dot(at_i, u[i]).sum()


def tensor_factors(x, s, pairs, alpha):
    """The displacement and the two factors of each pair's damped dipole tensor."""
    i, k, shift, _ = pairs
    v = x[k] + shift - x[i]
    r = dot(v, v).sqrt()
    bn, rr = bn_factors(r, alpha, 3)
    s3, s5, _ = thole_factors(r, s, i, k)
    return v, bn[1] - (1 - s3) * rr[1], bn[2] - (1 - s5) * rr[2]


def dipole_field(u, pairs, tensor):
    i, k, _, _ = pairs
    v, a, b = tensor
    out = torch.zeros_like(u)
    out.index_add_(0, i, -a[:, None] * u[k] + (b * dot(u[k], v))[:, None] * v)
    out.index_add_(0, k, -a[:, None] * u[i] + (b * dot(u[i], v))[:, None] * v)
    return out


def splines(w):
    """Values and first two derivatives of the five order-5 splines at offset w."""
    def values(order):
        m = [1 - w, w]
        for n in range(3, order + 1):
            new = []
            for j in range(n):      # M_n(w + n - 1 - j): node 0 is the farthest behind
                u = w + (n - 1 - j)
                left = m[j - 1] if j >= 1 else torch.zeros_like(w)
                right = m[j] if j < n - 1 else torch.zeros_like(w)
                new.append((u * left + (n - u) * right) / (n - 1))
            m = new
        return m

    def less(m):
        return [(m[j - 1] if j >= 1 else 0 * w) - (m[j] if j < len(m) else 0 * w) for j in range(len(m) + 1)]

    return torch.stack([torch.stack(values(5), -1), torch.stack(less(values(4)), -1),
                        torch.stack(less(less(values(3))), -1)])


class Mesh:
    """Order-5 smooth particle-mesh Ewald on a box and mesh."""

    def __init__(self, edges, mesh, alpha):
        self.edges, self.mesh = t64(edges), [int(m) for m in mesh]
        self.k = t64(self.mesh)
        mods, freq = [], []
        nodes = splines(torch.zeros((), dtype=torch.float64))[0].tolist()
        for n in self.mesh:
            j = np.arange(n)
            y = sum(c * np.exp(2j * np.pi * j * (q + 1) / n) for q, c in enumerate(nodes))
            b = np.abs(y) ** 2
            for m in range(n):
                if b[m] < 1e-7:
                    b[m] = 0.5 * b[1] if m == 0 else 0.5 * b[m - 1] if m == n - 1 else 0.5 * (b[m - 1] + b[m + 1])
            h = np.where(j > n // 2, j - n, j) * np.pi / n
            far = np.pi * np.arange(1, 51)
            with np.errstate(all="ignore"):
                up, down = h[:, None] / (h[:, None] + far), h[:, None] / (h[:, None] - far)
                zeta = (1 + (up ** 10 + down ** 10).sum(1)) / (1 + (up ** 5 + down ** 5).sum(1))
            mods.append(t64(b * zeta ** 2))
            freq.append(t64(np.where(j >= (n + 1) // 2, j - n, j)))
        f = [q / e for q, e in zip(freq, self.edges)]
        s2 = (f[2] ** 2)[:, None, None] + (f[1] ** 2)[None, :, None] + (f[0] ** 2)[None, None, :]
        bb = mods[2][:, None, None] * mods[1][None, :, None] * mods[0][None, None, :]
        term = -(math.pi / alpha) ** 2 * s2
        s2[0, 0, 0] = 1.0
        self.influence = torch.where(term > -50.0, torch.exp(term) / (s2 * math.pi * self.edges.prod() * bb), 0.0)
        self.influence[0, 0, 0] = 0.0

    def place(self, x):
        """Mesh points (n, 125) and the splines of each axis."""
        w = x / self.edges
        f = (w - torch.floor(w.detach() + 0.5) + 0.5) * self.k
        cell = torch.floor(f.detach())
        at = (cell[:, :, None] - 4 + torch.arange(5, device=DEV)) % self.k[None, :, None]
        at = at.long()
        nx, ny, _ = self.mesh
        flat = (at[:, 2, :, None, None] * ny + at[:, 1, None, :, None]) * nx + at[:, 0, None, None, :]
        return flat.reshape(len(x), 125), splines(f - cell)

    def weights(self, spl, q, d, Q):
        """(n, 125) mesh charges of multipoles (any of them None)."""
        c = self.k / self.edges
        x, y, z = spl[:, :, 0], spl[:, :, 1], spl[:, :, 2]
        out = 0.0
        def add(v, a, b, e):
            return v[:, None, None, None] * z[e][:, :, None, None] * y[b][:, None, :, None] * x[a][:, None, None, :]
        if q is not None:
            out = out + add(q, 0, 0, 0)
        if d is not None:
            out = out + add(c[0] * d[:, 0], 1, 0, 0) + add(c[1] * d[:, 1], 0, 1, 0) + add(c[2] * d[:, 2], 0, 0, 1)
        if Q is not None:
            for a in range(3):
                for b in range(a, 3):
                    order = [0, 0, 0]
                    order[a] += 1
                    order[b] += 1
                    out = out + add((2 if a != b else 1) / 3.0 * c[a] * c[b] * Q[:, a, b], *order)
        return out.reshape(len(spl[0]), 125)

    def potential(self, flat, weights):
        nx, ny, nz = self.mesh
        g = torch.zeros(nx * ny * nz, dtype=torch.float64, device=DEV).index_add(0, flat.reshape(-1), weights.reshape(-1))
        g = torch.fft.fftn(g.reshape(nz, ny, nx)) * self.influence
        return (torch.fft.ifftn(g).real * (nx * ny * nz)).reshape(-1)

    def field_of_dipoles(self, flat, spl, u):
        """Minus the gradient of the potential of dipoles u at every atom."""
        phi = self.potential(flat, self.weights(spl, None, u, None))[flat].reshape(-1, 5, 5, 5)
        c = self.k / self.edges
        x, y, z = spl[:, :, 0], spl[:, :, 1], spl[:, :, 2]
        part = lambda a, b, e: torch.einsum("nzyx,nx,ny,nz->n", phi, x[a], y[b], z[e])  # noqa: E731
        return -torch.stack([c[0] * part(1, 0, 0), c[1] * part(0, 1, 0), c[2] * part(0, 0, 1)], 1)


def electrostatics(x, local, inputs, use=None, vacuum=False, polar=True, lam_real=None):
    """[real, self, reciprocal] permanent energies, [real, self, reciprocal] polarization
    energies, and a function of x and the multipoles whose gradient is the polarization
    energy's; of the atoms in use, in the periodic box or alone in vacuum."""
    s, p = inputs["system"], inputs["params"]
    alpha = 0.0 if vacuum else p.ewald_alpha
    if use is not None:
        x, local = x[use], local[use]
        at = use.cpu().numpy()
        s = Part(s, at)
    pol = t64(s.polarizability)
    if vacuum:
        n = len(x)
        i, k = torch.triu_indices(n, n, 1, device=DEV)
        pairs = (i, k, torch.zeros(len(i), 3, device=DEV, dtype=torch.float64), torch.ones_like(i, dtype=torch.bool))
    else:
        pairs = inputs["real_pairs"] if use is None else pairs_within(x.detach(), p.box, p.ewald_cutoff)
    mult = global_multipoles(x, local)
    q, d, Q = mult
    el = p.electric
    real = el * permanent_real(x, mult, pairs, alpha, lam_real)
    zero = torch.zeros((), dtype=torch.float64, device=DEV)
    own = recip = zero
    if not vacuum:
        a2 = 2 * alpha * alpha
        own = -el * alpha / math.sqrt(math.pi) * (q * q + a2 * (dot(d, d) / 3 + 2 * a2 * (Q * Q).sum((1, 2)) / 45)).sum()
        mesh = inputs["mesh"]
        flat, spl = mesh.place(x)
        weights = mesh.weights(spl, q, d, Q)
        phi = mesh.potential(flat, weights)
        recip = 0.5 * el * (phi[flat] * weights).sum()
    if not polar:
        return (real, own, recip), (zero, zero, zero), zero
    a3 = 4.0 / 3.0 * alpha ** 3 / math.sqrt(math.pi)

    # With every p and d scale zero inside a molecule the two dipole sets are one.
    def source(u):
        """u . (real, self, reciprocal) parts of the permanent field."""
        parts = [field_dot(x, mult, u, s, pairs, alpha), zero, zero]
        if not vacuum:
            parts[1] = a3 * dot(u, d).sum()
            parts[2] = -(phi[flat] * mesh.weights(spl, None, u, None)).sum()
        return parts

    u = torch.zeros_like(x).requires_grad_(True)
    E = torch.autograd.grad(sum(source(u)), u, retain_graph=True)[0]
    with torch.no_grad():
        tensor = tensor_factors(x, s, pairs, alpha)
        if not vacuum:
            spl_now = spl.detach()

        def matrix(v):
            out = v / pol[:, None] - dipole_field(v, pairs, tensor) - a3 * v
            return out if vacuum else out - mesh.field_of_dipoles(flat, spl_now, v)

        u = pol[:, None] * E
        r = E - matrix(u)
        z = pol[:, None] * r
        v, rz = z, (r * z).sum()
        for _ in range(200):
            if float((r * r).sum()) <= 1e-26 * float((E * E).sum()):
                break
            av = matrix(v)
            step = rz / (v * av).sum()
            u, r = u + step * v, r - step * av
            z = pol[:, None] * r
            new = (r * z).sum()
            v, rz = z + new / rz * v, new
    parts = [-0.5 * el * e for e in source(u)]
    vv, a, b = tensor_factors(x, s, pairs, alpha)
    i, k = pairs[0], pairs[1]
    bent = 2 * (-a * dot(u[i], u[k]) + b * dot(u[i], vv) * dot(u[k], vv)).sum()
    if not vacuum:
        w = mesh.weights(spl, None, u, None)
        bent = bent - (mesh.potential(flat, w)[flat] * w).sum()
    inputs["dipoles"] = u
    return (real, own, recip), tuple(parts), 2 * sum(parts) - 0.5 * el * bent


class Part:
    """The atoms of a system that take part."""

    def __init__(self, s, at):
        self.polarizability, self.pdamp, self.thole = s.polarizability[at], s.pdamp[at], s.thole[at]


def evaluate(system, params, xyz, soft=None, lam=1.0, elec=False, fit=False):
    """The outputs of one evaluation at these coordinates, as run() lays them out."""
    x = t64(xyz).requires_grad_(True)
    local = t64(system.multipole).requires_grad_(True)
    lam = t64(lam).requires_grad_(True)
    inputs = {"system": system, "params": params, "mesh": Mesh(params.box, params.grid(), params.ewald_alpha),
              "soft": np.zeros(len(xyz), dtype=bool) if soft is None else soft > 0,
              "vdw_pairs": pairs_within(x.detach(), params.box, params.vdw_cutoff + 0.6),
              "real_pairs": pairs_within(x.detach(), params.box, params.ewald_cutoff)}
    vdw = vdw_energy(x, inputs, lam)
    if not elec:
        perm, pol, bent = electrostatics(x, local, inputs)
        total = vdw + sum(perm) + bent
    else:
        # Below the polarization window (lambda < 0.75): the whole system's permanent terms
        # grow with the window's power as those without the soft atoms and of the soft atoms
        # in vacuum fade; polarization is that of the two parts.
        start = 0.4
        w = ((lam - start) / (1 - start)).clamp(min=0.0)
        power = w ** 3
        is_soft = torch.as_tensor(inputs["soft"], device=DEV)
        i, k = inputs["real_pairs"][:2]
        add = 2.0 * (1 - w) ** 2 * (lam > start)
        p1, _, _ = electrostatics(x, local, inputs, polar=False, lam_real=(is_soft[i] | is_soft[k], add, power))
        p2, pol2, bent2 = electrostatics(x, local, inputs, use=~is_soft)
        p3, pol3, bent3 = electrostatics(x, local, inputs, use=is_soft, vacuum=True)
        perm = (p1[0] + (1 - power) * p3[0], power * p1[1] + (1 - power) * p2[1], power * p1[2] + (1 - power) * p2[2])
        pol = tuple(a + b for a, b in zip(pol2, pol3))
        total = vdw + sum(perm) + bent2 + bent3
    terms = [vdw, sum(perm), sum(pol), *perm, *pol, vdw + sum(perm) + sum(pol)]
    out = {"terms": torch.stack([t.detach() for t in terms]).cpu().numpy()}
    if elec:
        d1 = torch.autograd.grad(total, lam, create_graph=True)[0]
        d2 = torch.autograd.grad(d1, lam, retain_graph=True)[0]
        out["dEdXdL"] = torch.autograd.grad(d1, x, retain_graph=True)[0].cpu().numpy()
        out["dEdL"] = np.array([d1.item(), d2.item()])
    if fit:
        # dE/dalpha at fixed damping: the polarization energy is stationary in the dipoles.
        u = inputs["dipoles"]
        a = t64(system.polarizability)
        out["dEdalpha"] = (-0.5 * params.electric * dot(u, u) / (a * a)).cpu().numpy()
        dM = torch.autograd.grad(sum(perm) + bent, local, retain_graph=True)[0]
        out["dEdM"] = dM.cpu().numpy()
    out["gradient"] = torch.autograd.grad(total, x)[0].cpu().numpy()
    return out


def shake(x0, x, m):
    """Sides restored by impulses along the old sides, to rounding."""
    x, x0, inv = x.reshape(-1, 3, 3).copy(), x0.reshape(-1, 3, 3), 1.0 / m.reshape(-1, 3)
    for _ in range(200):
        worst = 0.0
        for a, b, d in ((0, 1, ROH), (0, 2, ROH), (1, 2, RHH)):
            r, r0 = x[:, b] - x[:, a], x0[:, b] - x0[:, a]
            miss = (r * r).sum(1) - d * d
            worst = max(worst, np.abs(miss).max())
            g = (miss / (2 * (r * r0).sum(1) * (inv[:, a] + inv[:, b])))[:, None] * r0
            x[:, a] += g * inv[:, a, None]
            x[:, b] -= g * inv[:, b, None]
        if worst < 1e-14:
            break
    return x.reshape(-1, 3)


def rattle(xyz, vel):
    """Velocities without motion along the sides."""
    x, v, inv = xyz.reshape(-1, 3, 3), vel.reshape(-1, 3, 3), 1.0 / masses(3)
    sides = ((0, 1), (1, 2), (2, 0))
    e = [x[:, b] - x[:, a] for a, b in sides]
    e = [u / np.linalg.norm(u, axis=1)[:, None] for u in e]
    push = np.zeros((3, len(x), 3, 3))      # what a unit impulse along each side does
    for j, (a, b) in enumerate(sides):
        push[j, :, a] -= inv[a] * e[j]
        push[j, :, b] += inv[b] * e[j]
    rate = lambda y: np.stack([((y[:, b] - y[:, a]) * e[j]).sum(1) for j, (a, b) in enumerate(sides)], 1)  # noqa: E731
    K = np.stack([rate(push[j]) for j in range(3)], 2)
    t = np.linalg.solve(K, -rate(v)[..., None])[..., 0]
    return (v + np.einsum("nj,jnab->nab", t, push)).reshape(-1, 3)


def exact(case, seed):
    work = systems_of(case, seed)
    s, p = work[0]
    if case["kind"] == "batch":
        outs = [evaluate(a, b, a.xyz) for a, b in work]
        return {"terms": np.stack([o["terms"] for o in outs]), "gradient": np.concatenate([o["gradient"] for o in outs])}
    if case["kind"] == "md":
        x, v, m, dt = s.xyz, velocities(s.xyz, seed), masses(s.n_atoms)[:, None], 0.002
        a = -KCAL * evaluate(s, p, x)["gradient"] / m
        ep, ek = [], []
        for _ in range(case["steps"]):
            new = shake(x, x + dt * (v + 0.5 * dt * a), m[:, 0])
            v, x = (new - x) / dt, new
            o = evaluate(s, p, x)
            a = -KCAL * o["gradient"] / m
            v = rattle(x, v + 0.5 * dt * a)
            ep.append(o["terms"][9])
            ek.append(0.5 * (m * v * v).sum() / KCAL)
        return {"xyz": x, "velocities": v, "epot": np.array(ep), "ekin": np.array(ek)}
    if case["kind"] == "lambda":
        return evaluate(s, p, s.xyz, soft=soft_atoms(case, seed), lam=case["lam"], elec=True)
    out = evaluate(s, p, s.xyz, fit=case["kind"] == "fit")
    return {"terms": out["terms"]} if case["kind"] == "energy" else out
