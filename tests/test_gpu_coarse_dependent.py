"""The coarse correction where boxes have fewer free DOFs than modes, so that A_c
is singular: the modes that the others span are set aside.  Held as in
test_gpu_coarse_edges: the residual, and the iterations of the same preconditioned
CG restated with the pseudo-inverse of A_c (its P A_c^+ P^T is that of any modes
that span the space)."""
import numpy as np
import pytest
import scipy.linalg as sla
import scipy.sparse as sp

from lpm_cases import cube, dense_from_bsr, make_gpu, pkg, plate
from test_coarse_emulation_cpu import _pcg, _prolongation
from test_gpu_onchip import TOL, _held

capi = pkg.capi
pytestmark = pytest.mark.gpu

CASES = {"plate 21x25, automatic": (lambda: plate(21, 25), 0.0), "plate 17x19, automatic": (lambda: plate(17, 19), 0.0),
         "plate 13x13": (lambda: plate(13, 13), 0.7), "cube 7, automatic": (lambda: cube(7), 0.0),
         "cube 9, automatic": (lambda: cube(9), 0.0)}


@pytest.mark.parametrize("name", list(CASES))
def test_coarse_solve_with_dependent_modes(name):
    make, box = CASES[name]
    case = make()
    dim, xyz = case[0], case[1]
    g = make_gpu(*case)
    axis = dim - 1
    c = xyz[:, axis]
    mask = np.zeros((len(xyz), 3), np.int32)
    mask[c < c.min() + 1e-9, :dim] = 1
    mask[c > c.max() - 1e-9, axis] = 1
    g.set_mask(mask)
    g.set_preconditioner(capi.PRECOND_COARSE, box)
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
    b = (np.random.default_rng(9).standard_normal((g.n, dim)) * (1 - mask[:, :dim])).ravel()
    g.upload(capi.F_RESIDUAL, b)
    it, rr, st = g.solve(capi.PREC_MIXED, TOL)
    x = g.download(capi.F_DISP)
    A = dense_from_bsr(*g.pattern(), g.K_bsr(), g.n, dim).T
    g.close()

    P = _prolongation(dim, xyz, mask[:, :dim].ravel().astype(bool), box)
    Ac = np.asarray(P.T @ (P.T @ A.T).T)
    free = np.diag(Ac) > 1e-12 * np.diag(Ac).max()
    assert np.linalg.matrix_rank(Ac, tol=1e-11 * np.abs(Ac).max()) < free.sum()
    inv = sla.pinvh(0.5 * (Ac + Ac.T), rtol=1e-11)
    Ps, Dinv = sp.csr_matrix(P), 1.0 / np.diag(A)
    _, ite = _pcg(A, b, lambda v: Dinv * v + Ps @ (inv @ (Ps.T @ v)), tol=TOL)
    r, bound = _held(A, b, x)
    print("[coarse dependent] %s: %d coarse DOFs, %d iterations (%d restated), residual %.2e of %.2e" % (
        name, len(Ac), it, ite, r, bound))
    assert st == capi.OK and r <= bound
    assert abs(it - ite) <= 0.1 * ite + 10
