"""Timed cases of the load-step library, each one pass through its public entry points.

A case is a dict of plain values with a "kind":

  step     one load step from a stored state (Lattice.load_step), positions and internal forces read back
  damage   one load step of the softening law with its damage rounds (static solver, eliminated tangent)
  cycle    one fatigue cycle of a compact-tension plate (Lattice.fatigue_cycle)
  j2       one plastic load step of a polycrystal with two tangent directions carried along
  adjoint  one backward step at a converged state (Lattice.backward_step)
  tangent  force pass, tangent assembly and one product with it (update, assemble, apply_operator)
  setup    bond search and creation of the device lattice (find_bonds, Lattice)

A pass that moves the lattice starts from a device checkpoint (the way LoadHistory replays a segment), so that it can be
repeated on one state.  Sizes and materials are those of the repository's configurations, tests and benchmark; the seed
varies the elastic constants, the load and the random draws of the material.
"""
import math

import numpy as np
import torch

import __graft_entry__

_pkg = __graft_entry__.load_package()
capi, lat = _pkg.capi, _pkg.lattice

PREC = {"fp64": capi.PREC_FP64, "mixed": capi.PREC_MIXED}
OPERATOR = {"assembled": capi.OPERATOR_ASSEMBLED, "free": capi.OPERATOR_MATRIX_FREE}
PRECOND = {"jacobi": capi.PRECOND_JACOBI, "coarse": capi.PRECOND_COARSE}
LATTICE = {"hex": lat.HEXAGON2D, "notched": lat.HEXAGON2D, "sc": lat.SIMPLECUBIC3D}
NEIGHBOURS = {"hex": 12, "notched": 12, "sc": 18, "ct": 12, "bcc": 14}
BLOCKS = {"hex": 31, "notched": 31, "sc": 61, "ct": 31, "bcc": 41}  # blocks of an interior row of the tangent
SPACING = {"hex": 0.5, "notched": 0.1, "sc": 0.2}
STEEL, ALUMINIUM, TITANIUM = (200e3, 0.3), (69e3, 0.3), (110e3, 0.34)
# Newton to 1e-8, as parity studies run it: internal forces then no longer hang on where the last linear solve stopped
NEWTON = dict(max_iter=60, tol=1e-8)


def listed():
    return [
        # the smallest call: the 40 x 40-cell plate of the isoelasticity example, the plain FP64 form with its defaults
        {"name": "plate41_fp64", "kind": "step", "lattice": "hex", "nx": 41, "ny": 41, "nz": 1, "precision": "fp64",
         "operator": "assembled"},
        # a small cube, as convergence studies and the tests run it
        {"name": "cube21_mixed", "kind": "step", "lattice": "sc", "nx": 21, "ny": 21, "nz": 21, "precision": "mixed",
         "operator": "assembled"},
        # the full-size single-edge-notched plate, one elastic step
        {"name": "notched201x401_mixed", "kind": "step", "lattice": "notched", "nx": 201, "ny": 401, "nz": 1,
         "precision": "mixed", "operator": "assembled"},
        # a ragged bar in the plain FP64 form, between the persistent loop's sizes and the largest cube
        {"name": "bar37x41x53_fp64", "kind": "step", "lattice": "sc", "nx": 37, "ny": 41, "nz": 53,
         "precision": "fp64", "operator": "assembled"},
        # a cube of a quarter of a million particles without an assembled operator
        {"name": "cube61_free", "kind": "step", "lattice": "sc", "nx": 61, "ny": 61, "nz": 61, "precision": "mixed",
         "operator": "free"},
        # the headline: the 100^3-cell cube, mixed precision
        {"name": "cube101_mixed", "kind": "step", "lattice": "sc", "nx": 101, "ny": 101, "nz": 101,
         "precision": "mixed", "operator": "assembled"},
        # damage rounds of a notched plate (softening bonds, Weibull strengths), with the coarse preconditioner
        {"name": "softening61x121_coarse", "kind": "damage", "nx": 61, "ny": 121, "precond": "coarse"},
        # one cycle of the compact-tension specimen at half the full plate's width
        {"name": "fatigue_w20_mixed", "kind": "cycle", "width": 20.0, "precond": "jacobi"},
        # one plastic step of a polycrystal with its two sensitivities
        {"name": "polycrystal24_tangents", "kind": "j2", "cells": 24, "grains": 8},
        # gradient of a reaction with respect to every bond's constants
        {"name": "adjoint41", "kind": "adjoint", "nx": 41, "ny": 41, "nz": 41},
        # a program that runs its own Krylov method: force pass, assembly, one product
        {"name": "tangent51_mixed", "kind": "tangent", "lattice": "sc", "nx": 51, "ny": 51, "nz": 51,
         "precision": "mixed"},
        # a new lattice: bond search, opposite bonds, pattern, layout
        {"name": "setup51", "kind": "setup", "nx": 51, "ny": 51, "nz": 51},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "damage", "cycle", "j2", "adjoint", "tangent", "setup"])
    if kind in ("step", "tangent"):
        lattice = rng.choice(["hex", "notched", "sc", "sc"])
        case = {"kind": kind, "lattice": lattice, "precision": rng.choice(["fp64", "mixed"])}
        if lattice == "sc":
            edge = _log_int(rng, 9, 70)
            case.update(nx=edge, ny=max(7, edge + rng.randint(-4, 4)), nz=max(7, edge + rng.randint(-4, 6)))
        else:
            edge = _log_int(rng, 21, 221)
            case.update(nx=edge, ny=2 * edge - rng.randint(0, edge // 2), nz=1)
        if kind == "step":
            case["operator"] = rng.choice(["assembled", "assembled", "free"])
        return case
    if kind == "damage":
        nx = _log_int(rng, 31, 81)
        return {"kind": kind, "nx": nx, "ny": 2 * nx - rng.randint(0, 9),
                "precond": rng.choice(["jacobi", "coarse"]) if nx <= 45 else "coarse"}
    if kind == "cycle":
        return {"kind": kind, "width": round(math.exp(rng.uniform(math.log(5.0), math.log(25.0))), 2),
                "precond": rng.choice(["jacobi", "coarse"])}
    if kind == "j2":
        return {"kind": kind, "cells": _log_int(rng, 9, 30), "grains": rng.randint(2, 12)}
    edge = _log_int(rng, 9, 61)
    return {"kind": kind, "nx": edge, "ny": max(7, edge + rng.randint(-3, 3)), "nz": max(7, edge + rng.randint(-3, 3))}


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return np.random.default_rng([20261203, int(seed)])


def _points(case, kind="sc"):
    """Particles, spacing and bond filter of a plate or a cube."""
    a = SPACING[kind]
    if kind == "sc":
        return lat.sc_cuboid(case["nx"], case["ny"], case["nz"], a), a
    return lat.hex_plate(case["nx"], case["ny"], a), a


def _crack(xyz, a, ny):
    """Height and tip of the notched plate's edge crack (sent_plate's rule, 0.3 of the width)."""
    return (ny // 2 - 0.5) * a * math.sqrt(3.0) / 2.0, xyz[:, 0].min() + 0.3 * (xyz[:, 0].max() - xyz[:, 0].min())


def _material(rng, E, nu):
    return E * rng.uniform(0.9, 1.1), nu * rng.uniform(0.9, 1.1)


def _body(case, kind, rng, constants):
    """(xyz, p1, p2, layer, Kn, Tv, cell) of a plate or a cube with the seed's elastic constants."""
    xyz, a = _points(case, kind)
    cell = lat.UnitCell(LATTICE[kind], a / 2)
    p1, p2, layer = capi.find_bonds(xyz, cell)
    if kind == "notched":
        y0, tip = _crack(xyz, a, case["ny"])
        p1, p2, layer = lat.precrack(xyz, p1, p2, layer, y0, tip)
    E, nu = _material(rng, *constants)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(E, nu, plane_stress=cell.dim == 2, layout="row"))
    return xyz, p1, p2, layer, Kn, Tv, cell


def _lattice(xyz, p1, p2, layer, Kn, Tv, cell):
    return capi.Lattice(cell.dim, xyz, p1, p2, layer, Kn, Tv, cell.particle_volume, cell.nneighbors)


def _faces(xyz, dim):
    c = xyz[:, dim - 1]
    return np.where(c < c.min() + 1e-9)[0], np.where(c > c.max() - 1e-9)[0]


def _tension(g, xyz, dim, du):
    """Uniaxial tension: a plate rolls on its lower edge, a cube is clamped at its lower face."""
    bottom, top = _faces(xyz, dim)
    gb, gt = g.add_group(bottom), g.add_group(top)
    if dim == 2:
        return [("disp", gb, 1, 0.0), ("disp", g.add_group(bottom[:1]), 0, 0.0), ("disp", gt, 1, du)]
    return [("disp", gb, 0, 0.0), ("disp", gb, 1, 0.0), ("disp", gb, 2, 0.0), ("disp", gt, 2, du)]


def _step_kind(case):
    return case.get("lattice", "sc")


def _step_load(case, rng, xyz, dim):
    """Top displacement of one load step: about 1e-4 of a cube's height, 5e-4 of a plate's."""
    c = xyz[:, dim - 1]
    return (1e-4 if dim == 3 else 5e-4) * (c.max() - c.min()) * rng.uniform(0.8, 1.2)


def _checked(r):
    if r["status"] != capi.OK:
        raise RuntimeError("load step did not converge: %s" % (r,))
    return r


def prepare(case, seed):
    rng = _rng(seed)
    return globals()["_prepare_" + case["kind"]](case, rng)


def _prepare_step(case, rng):
    kind = _step_kind(case)
    body = _body(case, kind, rng, STEEL if kind == "sc" else ALUMINIUM)
    xyz, dim = body[0], body[-1].dim
    g = _lattice(*body)
    g.set_operator(OPERATOR[case["operator"]])
    bcs = _tension(g, xyz, dim, _step_load(case, rng, xyz, dim))
    g.update()
    return {"kind": "step", "g": g, "bcs": bcs, "start": g.checkpoint_save(), "precision": PREC[case["precision"]]}


def _prepare_damage(case, rng):
    body = _body(case, "notched", rng, ALUMINIUM)
    xyz, p1, p2, layer = body[:4]
    g = _lattice(*body)
    g.set_law(capi.LAW_SOFTENING, [3.0, 1.0e-3])
    scrit = lat.weibull_draws(p1, p2, 10.0, 1.2e-3, int(rng.integers(1 << 30)))
    g.upload(capi.B_SCRIT, scrit[g.bond_perm])
    g.set_preconditioner(PRECOND[case["precond"]])
    # the increment in which the first bonds ahead of the notch soften: the tip strain grows with the root of the crack
    bcs = _tension(g, xyz, 2, 1.5e-4 * math.sqrt(201.0 / case["nx"]) * 0.1 * math.sqrt(0.75) * (case["ny"] - 1)
                   * rng.uniform(0.95, 1.05))
    g.update()
    return {"kind": "damage", "g": g, "bcs": bcs, "start": g.checkpoint_save()}


def _prepare_cycle(case, rng):
    a, L, f_max, R = 0.15, 0.3, 400.0 * math.sqrt(case["width"] / 40.0), 0.1
    xyz, p1, p2, layer, cell, info = lat.ct_specimen(case["width"], 0.4, a)
    E, nu = _material(rng, *TITANIUM)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(E, nu, plane_stress=True, layout="row"))
    n = len(xyz)
    g = _lattice(xyz, p1, p2, layer, Kn, Tv, cell)
    g.set_law(capi.LAW_FATIGUE_HCF, np.stack([rng.uniform(1.5e-4, 2.5e-4, n), rng.uniform(0.50, 0.65, n),
                                              np.full(n, 1.079), np.ones(n)], axis=1))
    (cx, cy_b), (_, cy_t) = info["holes"]
    near = (np.abs(xyz[:, 0] - cx) <= info["radius"]) & ((xyz[:, 1] >= cy_t) | (xyz[:, 1] <= cy_b))
    g.set_types(np.where(near, 4, 0).astype(np.int32), 4)  # the pin regions do not damage
    g.set_nonlocal(*capi.find_neighbors(xyz, 1.5 * L), L)
    g.set_preconditioner(PRECOND[case["precond"]])
    g.update()
    groups = lat.ct_groups(xyz, info, a)
    gm, gt, gb = g.add_group(groups["mid"]), g.add_group(groups["top"]), g.add_group(groups["bottom"])
    fixed = [("disp", gm, 1, 0.0), ("disp", gt, 0, 0.0), ("disp", gb, 0, 0.0)]
    low = R * f_max
    _checked(g.load_step(fixed + [("force", gt, 0.0, low, 0.0), ("force", gb, 0.0, -low, 0.0)],
                         precision=capi.PREC_MIXED, **NEWTON))
    return {"kind": "cycle", "g": g, "unit": fixed + [("force", gt, 0.0, 1.0, 0.0), ("force", gb, 0.0, -1.0, 0.0)],
            "loads": (low, f_max, low), "start": g.checkpoint_save()}


def _prepare_j2(case, rng):
    a = 0.2
    xyz, _ = lat.bcc_polycrystal(case["cells"], a, case["grains"], 11)
    cell = lat.UnitCell(lat.BCC3D, a * math.sqrt(3.0) / 4.0)
    xyz = xyz[lat.prune_weak(xyz, cell, 6)]
    p1, p2, layer = capi.find_bonds(xyz, cell)
    E, nu = _material(rng, *TITANIUM)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(E, nu, layout="row"))
    g = _lattice(xyz, p1, p2, layer, Kn, Tv, cell)
    g.set_law(capi.LAW_J2, [E, nu, 900.0 * rng.uniform(0.95, 1.05), 0.0, 1e3, 0.0, 0.0])
    g.update()
    z = xyz[:, 2]
    gb, gt = g.add_group(np.where(z < 0.1)[0]), g.add_group(np.where(z > z.max() - 0.1)[0])
    fixed = [("disp", gb, 0, 0.0), ("disp", gb, 1, 0.0), ("disp", gb, 2, 0.0)]
    height = z.max() - z.min()
    for _ in range(4):  # past yield: 0.8 % strain
        _checked(g.load_step(fixed + [("disp", gt, 2, 2e-3 * height)], precision=capi.PREC_MIXED, **NEWTON))
    return {"kind": "j2", "g": g, "bcs": fixed + [("disp", gt, 2, 1e-3 * height)], "start": g.checkpoint_save(),
            # d/d(yield stress) and d/d(hardening modulus)
            "directions": [[0, 0, 1, 0, 0, 0, 0], [0, 0, 0, 0, 1, 0, 0]]}


def _prepare_adjoint(case, rng):
    body = _body(case, "sc", rng, STEEL)
    xyz = body[0]
    g = _lattice(*body)
    bcs = _tension(g, xyz, 3, _step_load(case, rng, xyz, 3))
    g.update()
    _checked(g.load_step(bcs, precision=capi.PREC_MIXED, **NEWTON))
    reaction = np.zeros((g.n, 3))
    reaction[_faces(xyz, 3)[1], 2] = 1.0
    return {"kind": "adjoint", "g": g, "reaction": reaction}


def _moved(case, rng):
    """A strained, slightly uneven configuration and a vector to multiply."""
    kind = _step_kind(case)
    body = _body(case, kind, rng, STEEL if kind == "sc" else ALUMINIUM)
    xyz, dim = body[0], body[-1].dim
    x = xyz.copy()
    x[:, :dim] *= 1.0 + 1e-3 * rng.uniform(-1, 1, dim)
    x[:, :dim] += 1e-5 * SPACING[kind] * rng.standard_normal((len(x), dim))
    return body, x, rng.standard_normal(len(x) * dim)


def _prepare_tangent(case, rng):
    body, x, v = _moved(case, rng)
    return {"kind": "tangent", "g": _lattice(*body), "x": x, "v": v, "precision": PREC[case["precision"]]}


def _prepare_setup(case, rng):
    xyz, a = _points(case)
    n = len(xyz)
    order = np.argsort(np.arange(n) // 8 + 0.5 * rng.random(n))  # numbered by rows, not strictly along them
    xyz = xyz[order] + 1e-3 * a * rng.uniform(-1, 1, xyz.shape)
    return {"kind": "setup", "xyz": xyz, "cell": lat.UnitCell(lat.SIMPLECUBIC3D, a / 2),
            "material": _material(rng, *STEEL)}


# -------------------------------------------------------------------- passes
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_step(s):
    g = s["g"]
    g.checkpoint_restore(s["start"])
    _checked(g.load_step(s["bcs"], precision=s["precision"], **NEWTON))
    return {"xyz": g.download(capi.F_XYZ), "pin": g.download(capi.F_PIN)}


def _run_damage(s):
    g = s["g"]
    g.checkpoint_restore(s["start"])
    _checked(g.load_step(s["bcs"], solver=capi.SOLVER_STATIC_ELIMINATE, precision=capi.PREC_MIXED, **NEWTON))
    return {"xyz": g.download(capi.F_XYZ), "pin": g.download(capi.F_PIN), "damage": g.download(capi.B_BDAMAGE)}


def _run_cycle(s):
    g = s["g"]
    g.checkpoint_restore(s["start"])
    _checked(g.fatigue_cycle(s["unit"], *s["loads"], 1, 1000.0, precision=capi.PREC_MIXED, **NEWTON))
    return {"xyz": g.download(capi.F_XYZ), "pin": g.download(capi.F_PIN), "damage": g.download(capi.F_DAMAGE)}


def _run_j2(s):
    g = s["g"]
    g.checkpoint_restore(s["start"])
    g.tangent_begin(s["directions"], tol=1e-10)
    _checked(g.load_step(s["bcs"], precision=capi.PREC_MIXED, **NEWTON))
    out = {"xyz": g.download(capi.F_XYZ), "pin": g.download(capi.F_PIN), "state": g.state(),
           "dpin": [g.tangent_get(k, capi.T_PIN) for k in range(2)]}
    g.tangent_end()
    return out


def _run_adjoint(s):
    dkn, dtv, _, _ = s["g"].backward_step(dJdpin=s["reaction"], cg_tol=1e-12)
    return {"dkn": dkn, "dtv": dtv}


def _run_tangent(s):
    g = s["g"]
    g.upload(capi.F_XYZ, s["x"])
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_NONE)
    return {"product": g.apply_operator(s["v"], s["precision"]), "pin": g.download(capi.F_PIN)}


def _run_setup(s):
    xyz, cell = s["xyz"], s["cell"]
    p1, p2, layer = capi.find_bonds(xyz, cell)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(*s["material"], layout="row"))
    g = _lattice(xyz, p1, p2, layer, Kn, Tv, cell)
    cptr, cidx = g.pattern()
    bonds = g.bonds()
    g.close()
    return {"p1": p1, "p2": p2, "layer": layer, "cptr": cptr, "cidx": cidx, "opp": bonds["opp"]}


# ---------------------------------------------------------------------- work
def _size(case):
    """Particles, directed bonds, tangent blocks, dimension and particles along the longest edge."""
    kind = {"damage": "notched", "cycle": "ct", "j2": "bcc"}.get(case["kind"], _step_kind(case))
    if kind == "ct":
        edge = 1.25 * case["width"] / 0.15
        n = 1.2 / 1.25 * edge * edge / math.sqrt(0.75) * 0.9
    elif kind == "bcc":
        edge, n = 2 * case["cells"], 2 * case["cells"] ** 3
    else:
        edge = max(case["nx"], case["ny"], case.get("nz", 1))
        n = case["nx"] * case["ny"] * case.get("nz", 1)
    dim = 3 if kind in ("sc", "bcc") else 2
    return n, n * NEIGHBOURS[kind], n * BLOCKS[kind], dim, edge


def work(case):
    """Inputs and outputs once (per bond: partner, length, plastic stretch, damage, two constants; per particle:
    positions, loads, constraints, forces) and the multiplications of the solves, with about 5.5 iterations of
    conjugate gradients per particle along the longest edge."""
    n, nb, nblk, dim, edge = _size(case)
    state = 44 * nb + 120 * n
    product, cg = 2.0 * nblk * dim * dim, 5.5 * edge
    kind = case["kind"]
    if kind == "setup":
        return {"bytes": 24 * n + 16 * n + 16 * nb + 4 * nblk, "flops": 8.0 * nb}
    if kind == "tangent":
        return {"bytes": state + 16 * n * dim, "flops": 60.0 * nb + 20.0 * nblk + product}
    if kind == "adjoint":
        return {"bytes": state + 16 * nb, "flops": cg * 40.0 * nb}
    solves = {"step": 3, "damage": 20, "cycle": 6, "j2": 4}[kind]
    if kind == "damage" or case.get("precond") == "coarse":
        cg = 150.0
    flops = solves * cg * product + (2 * cg * 40.0 * nb if kind == "j2" else 0.0)
    return {"bytes": state + 48 * n + (16 * dim * n if kind == "j2" else 0), "flops": flops}


# --------------------------------------------------------- values in 64 bits
MOST_EXACT = 140_000  # particles; the pair search below takes n^2 distances


def _pairs(x, cut0, cut1):
    """Directed pairs closer than 1.01 cut1, by (i, j), layer 1 from 1.01 cut0 on: all distances, in chunks."""
    i, j, layer = [], [], []
    step = max(1, 200_000_000 // len(x))
    for at in range(0, len(x), step):
        d = sum((x[at:at + step, None, c] - x[None, :, c]) ** 2 for c in range(3)).sqrt_()
        near = d < 1.01 * cut1
        near[torch.arange(len(near)), torch.arange(at, at + len(near))] = False
        k = near.nonzero()
        i.append(k[:, 0] + at)
        j.append(k[:, 1])
        layer.append((d[near] >= 1.01 * cut0).long())
    return torch.cat(i), torch.cat(j), torch.cat(layer)


class _Body:
    """The lattice's internal forces and their derivative in plain torch, undamaged bonds:
    f_ij = 2 Kn dL_ij + 2 Tv sum of dL over the layer of i, Pin_i = sum of c_ij (f_ij + f_ji) / 2."""

    def __init__(self, case, kind, E, nu):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        a, self.dim = SPACING[kind], 3 if kind == "sc" else 2
        self.x0 = torch.tensor(_points(case, kind)[0], dtype=torch.float64, device=dev)
        self.n = len(self.x0)
        second = a * (math.sqrt(2.0) if kind == "sc" else math.sqrt(3.0))
        self.i, self.j, self.layer = _pairs(self.x0, a, second)
        if kind == "notched":
            y0, tip = _crack(self.x0, a, case["ny"])
            yi, yj = self.x0[self.i, 1], self.x0[self.j, 1]
            t = (y0 - yi) / torch.where(yi == yj, 1.0, yj - yi)
            xc = self.x0[self.i, 0] + t * (self.x0[self.j, 0] - self.x0[self.i, 0])
            keep = ~(((yi - y0) * (yj - y0) < 0) & (xc < tip))
            self.i, self.j, self.layer = self.i[keep], self.j[keep], self.layer[keep]
        if kind == "sc":
            C11, C12 = E * (1 - nu) / (1 + nu) / (1 - 2 * nu), E * nu / (1 + nu) / (1 - 2 * nu)
            C44, r = E / 2 / (1 + nu), a / 2
            kn, self.tv = (r * (C11 - C12 - C44), r * C44), r * (C12 - C44) / 18
        else:
            C11, C12 = E / (1 - nu * nu), E * nu / (1 - nu * nu)
            C44 = E / 2 / (1 + nu)
            k = math.sqrt(3.0) / 12 * (C11 - C12)
            kn, self.tv = (k, k), -math.sqrt(3.0) / 144 * C11 + math.sqrt(3.0) / 48 * C12
        self.kn = torch.where(self.layer == 0, kn[0], kn[1])
        self.seg = 2 * self.i + self.layer  # (owner, layer) of each bond
        key = self.i * self.n + self.j
        self.opp = torch.searchsorted(key, self.j * self.n + self.i)
        self.len0 = self._geometry(self.x0)[0]

    def _geometry(self, x):
        d = x[self.i] - x[self.j]
        length = d.square().sum(1).sqrt()
        return length, d / length[:, None]

    def _sum(self, index, count, values):
        return torch.zeros((count, *values.shape[1:]), dtype=torch.float64, device=values.device).index_add_(
            0, index, values)

    def _bond_force(self, dl):
        return 2 * self.kn * dl + 2 * self.tv * self._sum(self.seg, 2 * self.n, dl)[self.seg]

    def at(self, x):
        """Keeps the state x for pin() and product()."""
        self.length, self.c = self._geometry(x)
        self.dl = self.length - self.len0
        f = self._bond_force(self.dl)
        self.f = 0.5 * (f + f[self.opp])

    def pin(self):
        return self._sum(self.i, self.n, self.c * self.f[:, None])

    def product(self, v, turning=True):
        """dPin along v (n x 3); without `turning` the bond directions stay (the analytical tangent)."""
        u = v[self.i] - v[self.j]
        dd = (self.c * u).sum(1)
        df = self._bond_force(dd)
        y = self.c * (0.5 * (df + df[self.opp]))[:, None]
        if turning:
            y = y + (u - self.c * dd[:, None]) * (self.f / self.length)[:, None]
        return self._sum(self.i, self.n, y)

    def solve(self, g, free, tol):
        """H_ff y = g by conjugate gradients."""
        y, r = torch.zeros_like(g), g * free
        p, rr = r.clone(), r.square().sum()
        stop = tol * tol * rr
        for k in range(20 * self.n):
            if k % 16 == 0 and bool(rr <= stop):
                break
            q = self.product(p) * free
            alpha = rr / (p * q).sum().clamp_min(1e-300)
            y, r = y + alpha * p, r - alpha * q
            new = r.square().sum()
            p, rr = r + (new / rr.clamp_min(1e-300)) * p, new
        return y

    def equilibrium(self, du):
        """Positions under the tension of _tension with the top moved by du, and the free components."""
        c = self.x0[:, self.dim - 1]
        bottom, top = c < c.min() + 1e-9, c > c.max() - 1e-9
        free = torch.ones_like(self.x0)
        free[:, self.dim:] = 0.0
        free[top, self.dim - 1] = 0.0
        if self.dim == 3:
            free[bottom] = 0.0
        else:
            free[bottom, 1] = 0.0
            free[bottom.nonzero()[0, 0], 0] = 0.0
        x = self.x0.clone()
        x[top, self.dim - 1] += du
        self.at(x)
        for _ in range(12):
            pin = self.pin()
            if float((pin * free).norm()) <= 1e-11 * max(float(pin.norm()), 1e-300):
                break
            x = x + self.solve(-pin * free, free, 1e-9)
            self.at(x)
        return x, free


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("step", "adjoint", "tangent") or _size(case)[0] > MOST_EXACT:
        return None
    rng, lattice = _rng(seed), _step_kind(case)
    if kind == "tangent":
        E, nu = _material(rng, *(STEEL if lattice == "sc" else ALUMINIUM))
        body = _Body(case, lattice, E, nu)
        x0 = body.x0.cpu().numpy()
        x = x0.copy()  # as _moved
        x[:, :body.dim] *= 1.0 + 1e-3 * rng.uniform(-1, 1, body.dim)
        x[:, :body.dim] += 1e-5 * SPACING[lattice] * rng.standard_normal((len(x), body.dim))
        v = rng.standard_normal(len(x) * body.dim).reshape(len(x), body.dim)
        dev = body.x0.device
        body.at(torch.tensor(x, device=dev))
        v3 = torch.zeros_like(body.x0)
        v3[:, :body.dim] = torch.tensor(v, device=dev)
        y = body.product(v3, turning=False)[:, :body.dim]
        return {"product": y.reshape(-1).cpu().numpy(), "pin": body.pin().cpu().numpy()}
    E, nu = _material(rng, *(STEEL if lattice == "sc" else ALUMINIUM))
    body = _Body(case, lattice, E, nu)
    x, free = body.equilibrium(_step_load(case, rng, body.x0.cpu().numpy(), body.dim))
    if kind == "step":
        return {"xyz": x.cpu().numpy(), "pin": body.pin().cpu().numpy()}
    # the response is the top face's reaction: mu = c - lambda, H_ff lambda = (H c)_f
    c = body.x0[:, 2]
    weight = torch.zeros_like(x)
    weight[c > c.max() - 1e-9, 2] = 1.0
    mu = weight - body.solve(body.product(weight) * free, free, 1e-12)
    along = (body.c * (mu[body.i] - mu[body.j])).sum(1)
    stored = torch.argsort(2 * body.i + body.layer, stable=True)
    total = body._sum(body.seg, 2 * body.n, body.dl)[body.seg]
    return {"dkn": (body.dl * along)[stored].cpu().numpy(), "dtv": (total * along)[stored].cpu().numpy()}
