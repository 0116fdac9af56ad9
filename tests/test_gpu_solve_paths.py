"""Which kernel a solve runs in, and the solve in each: on chip (k_pcg_mixed,
k_pcg_fp64) with every number of slices to a block that changes the split of
its work, at grid barriers (k_mx_persistent, k_cg_persistent) past the on-chip
solves' limits, the graph loop's product on 32-bit columns.  A solve is held to
its stopping rule on the operator in FP64, |b - A x| <= tol |b| plus the
rounding of forming the residual, 1e-13 |A| |x|, and its iterations to the graph
loop's (5 % and four: the sums are folded in another order)."""
import numpy as np
import pytest

from lpm_cases import lat, make_gpu, pkg
from test_gpu_onchip import CASES, TOL

capi = pkg.capi
pytestmark = pytest.mark.gpu
MIXED, FP64 = capi.PREC_MIXED, capi.PREC_FP64


def _body(dim, size, window=0):
    """A plate or a box; numbered at random within windows of that many particles."""
    if dim == 2:
        cell, xyz = lat.UnitCell(lat.HEXAGON2D, 0.25), lat.hex_plate(*size, 0.5)
    else:
        cell, xyz = lat.UnitCell(lat.SIMPLECUBIC3D, 0.1), lat.sc_cuboid(*size, 0.2)
    rng, n = np.random.default_rng(4), len(xyz)
    if window:
        at = np.concatenate([a + rng.permutation(min(window, n - a)) for a in range(0, n, window)])
        xyz = xyz[at]
    p1, p2, layer = capi.find_bonds(xyz, cell)
    Kn, Tv = lat.bond_constants(cell, layer, cell.elastic_constants(69e3, 0.3, plane_stress=dim == 2, layout="row"))
    return dim, xyz, p1, p2, layer, Kn, Tv, cell


class System:
    def __init__(self, case, precond=None):
        dim, xyz = case[0], case[1]
        self.g = g = make_gpu(*case)
        c, axis = xyz[:, dim - 1], dim - 1
        mask = np.zeros((g.n, 3), np.int32)
        mask[c < c.min() + 1e-9, :dim] = 1
        mask[c > c.max() - 1e-9, axis] = 1
        g.set_mask(mask)
        if precond is not None:
            g.set_preconditioner(precond, 0.0)
        g.update()
        g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
        self.b = (np.random.default_rng(3).standard_normal((g.n, dim)) * (1 - mask[:, :dim])).ravel()
        cptr, cidx = g.pattern()
        rows = np.abs(g.K_bsr()).reshape(-1, dim * dim).sum(1)  # each block's entries, an upper bound of its share of |A|
        self.norm = np.add.reduceat(rows, cptr[:-1]).max()
        self.reach = np.abs(cidx - np.repeat(np.arange(g.n), np.diff(cptr))).max()

    def solve(self, precision, loop=capi.CG_LOOP_AUTO):
        """(iterations, persistent solves, on-chip solves) of one solve, held to its residual."""
        g = self.g
        g.set_cg_loop(loop)
        g.upload(capi.F_RESIDUAL, self.b)
        g.reset_stats()
        it, _, st = g.solve(precision, TOL)
        x, s = g.download(capi.F_DISP), g.stats()
        r = np.linalg.norm(self.b - np.ravel(g.apply_operator(x)))
        bound = TOL * np.linalg.norm(self.b) + 1e-13 * self.norm * np.linalg.norm(x)
        print("[paths] n %d, precision %d, loop %d: %d iterations, %d persistent, %d on chip, residual %.2e of %.2e" % (
            g.n, precision, loop, it, s["persistent_solves"], g.onchip_solves(), r, bound))
        assert st == capi.OK and s["mixed_fallbacks"] == 0 and r <= bound
        return it, s["persistent_solves"], g.onchip_solves()


def _like(it, graph):
    return abs(it - graph) <= 0.05 * graph + 4


@pytest.mark.parametrize("precision", [MIXED, FP64])
def test_edge_cases_run_on_chip(precision):
    """The systems of the on-chip tests do run there, the coarse correction too."""
    for name in CASES:
        s = System(CASES[name]())
        assert s.solve(precision)[1:] == (1, 1), name
        s.g.close()
    s = System(CASES["plate 40x60"](), capi.PRECOND_COARSE)
    assert s.solve(MIXED)[1:] == (1, 1)
    s.g.close()


# size: slices of the largest of 152 blocks
ON_CHIP_FP64 = {"plate 61x121": (2, (61, 121), 0),      # 2, seven warps, two blocks an SM
                "plate 91x105": (2, (91, 105), 0),      # 2
                "plate 120x120": (2, (120, 120), 0),    # 3
                "plate 140x170": (2, (140, 170), 0),    # 5
                "plate 190x190": (2, (190, 190), 0),    # 8, eight warps
                "plate 190x210": (2, (190, 210), 0),    # 9, twelve
                "plate 230x252": (2, (230, 252), 0),    # 12
                "plate 220x250 in windows": (2, (220, 250), 16384),  # 12, 9.9k columns: the tail blocks not kept
                "box 24x25x26": (3, (24, 25, 26), 0),   # 4
                "box 30x30x30": (3, (30, 30, 30), 0),   # 6
                "box 38x38x38": (3, (38, 38, 38), 0)}   # 12
ON_CHIP_MIXED = {"plate 61x121": (2, (61, 121), 0),     # 2, six warps, two blocks an SM
                 "box 12x13x14": (3, (12, 13, 14), 0),  # 1, seven
                 "box 35x35x35": (3, (35, 35, 35), 0),  # 9
                 "box 38x38x38": (3, (38, 38, 38), 0),  # 12
                 "box 41x41x41": (3, (41, 41, 41), 0)}  # 15


@pytest.mark.parametrize("name,precision", [(k, FP64) for k in ON_CHIP_FP64] + [(k, MIXED) for k in ON_CHIP_MIXED])
def test_on_chip_with_several_slices_a_block(name, precision):
    s = System(_body(*(ON_CHIP_FP64 if precision == FP64 else ON_CHIP_MIXED)[name]))
    it, persistent, on_chip = s.solve(precision)
    assert (persistent, on_chip) == (1, 1)
    graph, persistent, on_chip = s.solve(precision, capi.CG_LOOP_GRAPH)
    assert (persistent, on_chip) == (0, 0) and _like(it, graph)
    s.g.close()


@pytest.mark.parametrize("size,window,on_chip", [((190, 210), 10**9, 1),  # 9 slices, 28.0 columns a row
                                                 ((200, 230), 10**9, 0),  # 10, 28.1
                                                 ((200, 230), 4096, 1)])  # 10, 18.6
def test_fp64_solve_of_scattered_numberings(size, window, on_chip):
    """On chip in 2-D up to 26 columns a row where a block has more than nine
    slices (past that k_cg_persistent is the faster); the mixed solve always."""
    s = System(_body(2, size, window))
    it, persistent, here = s.solve(FP64)
    assert (persistent, here) == (1, on_chip)
    assert _like(it, s.solve(FP64, capi.CG_LOOP_GRAPH)[0])
    assert s.solve(MIXED)[1:] == (1, 1)
    s.g.close()


@pytest.mark.parametrize("dim,size,precision", [(2, (250, 245), FP64),    # 13 slices: k_cg_persistent
                                                (3, (40, 40, 40), FP64),  # 14
                                                (2, (345, 345), MIXED),   # 25: k_mx_persistent
                                                (3, (43, 43, 43), MIXED)])  # 17
def test_grid_barrier_solve_past_the_on_chip_limits(dim, size, precision):
    s = System(_body(dim, size))
    it, persistent, on_chip = s.solve(precision, capi.CG_LOOP_PERSISTENT)
    assert (persistent, on_chip) == (1, 0)
    graph, persistent, on_chip = s.solve(precision, capi.CG_LOOP_GRAPH)
    assert (persistent, on_chip) == (0, 0) and _like(it, graph)
    s.g.close()


@pytest.mark.parametrize("dim,size", [(2, (345, 345)), (3, (43, 43, 43))])
def test_grid_barrier_coarse_solve_past_the_on_chip_limits(dim, size):
    """k_mx_persistent with the coarse correction: its residual, and fewer
    iterations than without."""
    s = System(_body(dim, size), capi.PRECOND_COARSE)
    it, persistent, on_chip = s.solve(MIXED)
    assert (persistent, on_chip) == (1, 0)
    s.g.set_preconditioner(capi.PRECOND_JACOBI)
    assert it < 0.7 * s.solve(MIXED, capi.CG_LOOP_GRAPH)[0]
    s.g.close()


@pytest.mark.parametrize("dim,size", [(2, (190, 190)), (3, (33, 33, 33))])
def test_graph_loop_on_32_bit_columns(dim, size):
    """Columns further than 16 bits from their rows: the graph loop's FP32
    product on 32-bit columns, against the same solve on chip."""
    s = System(_body(dim, size, 10**9))
    assert s.reach > 32767
    it, persistent, on_chip = s.solve(MIXED)
    assert (persistent, on_chip) == (1, 1)
    graph, persistent, on_chip = s.solve(MIXED, capi.CG_LOOP_GRAPH)
    assert (persistent, on_chip) == (0, 0) and _like(it, graph)
    s.g.close()
