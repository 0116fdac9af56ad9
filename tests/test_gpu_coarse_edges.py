"""The coarse correction at the edges of its set-up and of its place in the
solve: fewer coarse DOFs than one step of the blocked inverse, a ragged last
step, one box, boxes whose DOFs are all eliminated, boxes cut by many blocks
of rows, particles numbered against their positions.  The solve is held to its
stopping rule on the operator in FP64, and its iterations to those of the same
preconditioned CG restated on the CPU with the exact inverse of A_c: 10% and
two reliable updates' worth (10) apart at most, the spread that restarting the
residual gives."""
import numpy as np
import pytest
import scipy.linalg as sla
import scipy.sparse as sp

from lpm_cases import cube, dense_from_bsr, make_gpu, pkg, plate
from test_coarse_emulation_cpu import _pcg, _prolongation
from test_gpu_onchip import TOL, _held, _renumbered

capi = pkg.capi
pytestmark = pytest.mark.gpu

# case, box edge, edge of the strip or slab of particles held in full (boxes with
# fewer free DOFs than modes, but some, are left out: A_c is singular there)
CASES = {
    "plate 9x9, one box": (lambda: plate(9, 9), 100.0, 0.0),           # 3 coarse DOFs
    "plate 13x13": (lambda: plate(13, 13), 0.9, 0.0),
    "plate 21x33": (lambda: plate(21, 33), 1.2, 0.0),
    "plate 33x33, boxes all held": (lambda: plate(33, 33), 0.95, 1.1),
    "plate 40x60": (lambda: plate(40, 60), 4.0, 0.0),
    "plate renumbered": (lambda: _renumbered(plate(27, 33), 5), 0.9, 0.0),
    "cube 5, one box": (lambda: cube(5), 100.0, 0.0),                  # 6 coarse DOFs
    "cube 8": (lambda: cube(8), 0.5, 0.0),
    "cube 12": (lambda: cube(12), 0.7, 0.6),
    "cube renumbered": (lambda: _renumbered(cube(9), 6), 0.7, 0.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_coarse_solve(name):
    make, box, held = CASES[name]
    case = make()
    dim, xyz = case[0], case[1]
    g = make_gpu(*case)
    axis = dim - 1
    c = xyz[:, axis]
    mask = np.zeros((len(xyz), 3), np.int32)
    mask[c < c.min() + 1e-9 + held, :dim] = 1
    mask[c > c.max() - 1e-9, axis] = 1
    g.set_mask(mask)
    g.set_preconditioner(capi.PRECOND_COARSE, box)
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
    b = np.random.default_rng(9).standard_normal((g.n, dim)) * (1 - mask[:, :dim])
    g.upload(capi.F_RESIDUAL, b.ravel())
    it, rr, st = g.solve(capi.PREC_MIXED, TOL)
    x = g.download(capi.F_DISP)
    A = dense_from_bsr(*g.pattern(), g.K_bsr(), g.n, dim).T
    g.close()
    b = b.ravel()

    fixed = mask[:, :dim].ravel().astype(bool)
    P = _prolongation(dim, xyz, fixed, box)
    Ac = np.asarray(P.T @ (P.T @ A.T).T)  # P^T A P
    inv = sla.pinvh(0.5 * (Ac + Ac.T), rtol=1e-11)
    Ps, Dinv = sp.csr_matrix(P), 1.0 / np.diag(A)
    _, ite = _pcg(A, b, lambda v: Dinv * v + Ps @ (inv @ (Ps.T @ v)), tol=TOL)
    r, bound = _held(A, b, x)
    print("[coarse edges] %s: %d coarse DOFs, %d iterations (%d restated), residual %.2e of a bound of %.2e"
          % (name, len(Ac), it, ite, r, bound))
    assert st == capi.OK and r <= bound
    assert abs(it - ite) <= 0.1 * ite + 10
