"""The matrix-free passes with one and with two lanes to a particle (chosen by
the number of particles and the precision) against the assembled products,
with the bounds of test_gpu_matrix_free.py: a ragged last warp, particles with
an odd number of bonds, damaged bonds."""
import numpy as np
import pytest

from lpm_cases import cube, make_gpu, pkg, plate, rel
from test_gpu_onchip import CASES

capi = pkg.capi
pytestmark = pytest.mark.gpu

SIZES = {"plate 4x3": CASES["plate 4x3"], "bar 2x3x11": CASES["bar 2x3x11"], "cube 12": lambda: cube(12),
         "plate 190x190 (FP64: one)": lambda: plate(190, 190), "cube 33 (FP64: one)": lambda: cube(33),
         "cube 69 (one)": lambda: cube(69)}


@pytest.mark.parametrize("name", list(SIZES))
def test_products_match_assembled_operator(name):
    g = make_gpu(*SIZES[name]())
    rng = np.random.default_rng(5)
    g.upload(capi.B_BDAMAGE, np.where(rng.random(g.nb) < 0.02, rng.random(g.nb), 0.0))
    g.update()
    v = np.tile(np.array([1.0, -0.5, 0.25])[:g.dim], g.n) + 1e-3 * rng.standard_normal(g.ndof)
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_NONE)
    y, y32 = g.apply_operator(v), g.apply_operator(v, capi.PREC_MIXED)
    g.set_operator(capi.OPERATOR_MATRIX_FREE)
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_NONE)
    e64, e32, e32a = rel(g.apply_operator(v), y), rel(g.apply_operator(v, capi.PREC_MIXED), y), rel(y32, y)
    print("[matrix-free lanes] %s: FP64 %.2e, FP32 %.2e (assembled FP32 %.2e)" % (name, e64, e32, e32a))
    assert e64 <= 1e-12 and e32 <= 2 * e32a + 1e-7
    g.close()
