"""The graph loop's vector kernels take four entries at a time: sizes of
every remainder, and less than one group of four blocks.  Each mixed solve is
held to its stopping rule on the operator in FP64 (as the on-chip ones)."""
import pytest

from lpm_cases import cube, pkg, plate
from test_gpu_onchip import CASES, _held, _solve

capi = pkg.capi
pytestmark = pytest.mark.gpu

# DOFs mod 4
SIZES = {"cube 3": (CASES["cube 3"], 1), "plate 4x3": (CASES["plate 4x3"], 2), "cube 5": (lambda: cube(5), 3),
         "bar 5x4x9": (CASES["bar 5x4x9"], 0), "plate 40x60": (lambda: plate(40, 60), 0)}


@pytest.mark.parametrize("name", list(SIZES))
def test_mixed_graph_solve(name):
    make, rest = SIZES[name]
    A, b, x, it, st, persistent = _solve(make(), capi.PREC_MIXED, loop=capi.CG_LOOP_GRAPH)
    r, bound = _held(A, b, x)
    print("[graph] %s: %d iterations, residual %.2e of a bound of %.2e" % (name, it, r, bound))
    assert len(b) % 4 == rest and st == capi.OK and persistent == 0
    assert r <= bound
