"""The on-chip CG solves (lpm_pcg.cu) at the edges of their layout: fewer rows
than one 32-row slice, a ragged last slice, every length of a slice's tail
of single blocks, one share of a slice's groups and many, blocks of one slice
and of several, particles numbered against their positions, one-sided bond
damage.  Each solve is held to its own stopping rule on the assembled
operator in FP64: |b - A x| <= tol |b|, plus the rounding of forming the
residual, 1e-13 |A| |x|."""
import numpy as np
import pytest

from lpm_cases import cube, dense_from_bsr, lat, make_gpu, pkg, plate

capi = pkg.capi
pytestmark = pytest.mark.gpu

TOL = 1e-10


def _renumbered(case, seed):
    dim, xyz, p1, p2, layer, Kn, Tv, cell = case
    new = np.random.default_rng(seed).permutation(len(xyz))  # new number of each particle
    x = np.empty_like(xyz)
    x[new] = xyz
    q1, q2 = new[p1].astype(np.int32), new[p2].astype(np.int32)
    order = np.lexsort((q2, q1))
    return dim, x, q1[order], q2[order], layer[order], Kn[order], Tv[order], cell


def _bar(nx, ny, nz):
    cell = lat.UnitCell(lat.SIMPLECUBIC3D, 0.1)
    xyz = lat.sc_cuboid(nx, ny, nz, 0.2)
    p1, p2, layer = lat.find_bonds(xyz, cell)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(200e3, 0.3, layout="row"))
    return 3, xyz, p1, p2, layer, Kn, Tv, cell


CASES = {
    "plate 4x3": lambda: plate(4, 3),      # 11 rows, one slice
    "plate 11x3": lambda: plate(11, 3),    # 32 rows
    "plate 11x3 + 1": lambda: plate(7, 5),  # 33 rows: a last slice of one row
    "plate 13x29": lambda: plate(13, 29),
    "plate 40x60": lambda: plate(40, 60),
    "plate renumbered": lambda: _renumbered(plate(17, 23), 5),
    "cube 3": lambda: cube(3),
    "bar 2x3x11": lambda: _bar(2, 3, 11),
    "bar 5x4x9": lambda: _bar(5, 4, 9),
    "cube 12": lambda: cube(12),
    "cube renumbered": lambda: _renumbered(cube(9), 6),
}


def _solve(case, precision, damage=False, loop=capi.CG_LOOP_AUTO, maxit=-1):
    dim, xyz, p1, p2, layer, Kn, Tv, cell = case
    g = make_gpu(dim, xyz, p1, p2, layer, Kn, Tv, cell)
    rng = np.random.default_rng(9)
    axis = dim - 1
    c = xyz[:, axis]
    mask = np.zeros((len(xyz), 3), np.int32)
    mask[c < c.min() + 1e-9, :dim] = 1
    mask[c > c.max() - 1e-9, axis] = 1
    g.set_mask(mask)
    if damage:
        g.upload(capi.B_BDAMAGE, np.where(rng.random(g.nb) < 0.05, 0.5 * rng.random(g.nb), 0.0))
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
    b = rng.standard_normal((g.n, dim)) * (1 - mask[:, :dim])
    g.upload(capi.F_RESIDUAL, b.ravel())
    g.set_cg_loop(loop)
    g.reset_stats()
    it, rr, st = g.solve(precision, TOL, maxit=maxit)
    x, on_chip = g.download(capi.F_DISP), g.stats()["persistent_solves"]
    A = dense_from_bsr(*g.pattern(), g.K_bsr(), g.n, dim).T
    g.close()
    return A, b.ravel(), x, it, st, on_chip


def _held(A, b, x):
    bound = TOL * np.linalg.norm(b) + 1e-13 * np.abs(A).sum(1).max() * np.linalg.norm(x)
    return np.linalg.norm(b - A @ x), bound


@pytest.mark.parametrize("name", list(CASES))
def test_mixed_solve_on_chip(name):
    A, b, x, it, st, on_chip = _solve(CASES[name](), capi.PREC_MIXED)
    r, bound = _held(A, b, x)
    print("[on chip] %s: %d iterations, residual %.2e of a bound of %.2e" % (name, it, r, bound))
    assert st == capi.OK and on_chip == 1
    assert r <= bound


@pytest.mark.parametrize("name", list(CASES))
def test_fp64_solve_on_chip(name):
    _solve(CASES["cube 12"](), capi.PREC_MIXED)  # other data left in the SMs' shared memory
    A, b, x, it, st, on_chip = _solve(CASES[name](), capi.PREC_FP64)
    r, bound = _held(A, b, x)
    print("[on chip] %s: %d FP64 iterations, residual %.2e of a bound of %.2e" % (name, it, r, bound))
    assert st == capi.OK and on_chip == 1
    assert r <= bound


def test_fp64_solve_stops_at_the_limit():
    """At a limit of 7 iterations, the graph loop's iterate to rounding."""
    case = plate(17, 23)
    _, b, x, it, st, on_chip = _solve(case, capi.PREC_FP64, maxit=7)
    _, _, xg, itg, stg, _ = _solve(case, capi.PREC_FP64, maxit=7, loop=capi.CG_LOOP_GRAPH)
    assert on_chip == 1 and it == itg == 7 and st == stg == capi.NOT_CONVERGED
    assert np.abs(x - xg).max() <= 1e-13 * np.abs(xg).max() * np.linalg.norm(b)


@pytest.mark.parametrize("precision", [capi.PREC_MIXED, capi.PREC_FP64])
def test_handles_of_two_sizes_in_turn(precision):
    """A small system's solve between two of a larger one: the launch limits
    are the kernel's, not the handle's."""
    big, small = make_gpu(*plate(40, 60)), make_gpu(*plate(5, 5))
    res = []
    for g in (big, small, big):
        mask = np.zeros((g.n, 3), np.int32)
        mask[:9, :2] = 1
        g.set_mask(mask)
        g.update()
        g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
        b = np.random.default_rng(g.n).standard_normal((g.n, 2)) * (1 - mask[:, :2])
        g.upload(capi.F_RESIDUAL, b.ravel())
        g.reset_stats()
        assert g.solve(precision, TOL)[2] == capi.OK and g.stats()["persistent_solves"] == 1
        res.append(g.download(capi.F_DISP))
    assert np.array_equal(res[0], res[2])
    big.close()
    small.close()


def test_mixed_solve_on_chip_with_damage():
    """A few bonds damaged on one side: A is no longer symmetric, and CG on it
    takes the graph loop's iterations to the same residual."""
    case = plate(13, 17)
    A, b, x, it, st, on_chip = _solve(case, capi.PREC_MIXED, damage=True)
    _, _, _, itg, stg, _ = _solve(case, capi.PREC_MIXED, damage=True, loop=capi.CG_LOOP_GRAPH)
    assert np.abs(A - A.T).max() > 1e-6 * np.abs(A).max()
    assert on_chip == 1 and st == stg
    if st == capi.OK:
        r, bound = _held(A, b, x)
        assert r <= bound and abs(it - itg) <= 0.05 * itg + 4


@pytest.mark.parametrize("nx,ny", [(190, 190), (215, 215), (240, 240), (275, 275), (336, 336)])
def test_mixed_solve_on_chip_of_many_slices_a_block(nx, ny):
    """8, 10, 12, 16 and 24 slices in the largest block: a block's threads and
    the warps of a slice change between them."""
    g = make_gpu(*plate(nx, ny))
    xyz = g.download(capi.F_XYZ)
    mask = np.zeros((g.n, 3), np.int32)
    mask[xyz[:, 1] < xyz[:, 1].min() + 1e-9, :2] = 1
    mask[xyz[:, 1] > xyz[:, 1].max() - 1e-9, 1] = 1
    g.set_mask(mask)
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
    b = (np.random.default_rng(3).standard_normal((g.n, 2)) * (1 - mask[:, :2])).ravel()
    g.upload(capi.F_RESIDUAL, b)
    g.reset_stats()
    it, rr, st = g.solve(capi.PREC_MIXED, TOL)
    x = g.download(capi.F_DISP)
    cptr, _ = g.pattern()
    rows = np.abs(g.K_bsr()).reshape(-1, 4).sum(1)  # each block's entries, an upper bound of its share of |A|
    norm = np.add.reduceat(rows, cptr[:-1]).max()
    r = np.linalg.norm(b - np.ravel(g.apply_operator(x)))
    bound = TOL * np.linalg.norm(b) + 1e-13 * norm * np.linalg.norm(x)
    print("[on chip] plate %dx%d: %d iterations, residual %.2e of a bound of %.2e" % (nx, ny, it, r, bound))
    assert st == capi.OK and g.stats()["persistent_solves"] == 1 and r <= bound
    g.close()
