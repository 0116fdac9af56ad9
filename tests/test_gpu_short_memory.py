"""The assembly's bond records are memory that only makes it faster: where the
rest of a solve does not fit beside them, they are given back, and the solve
and later assemblies go on as without them, to the same bits of K."""
import numpy as np
import pytest
import torch

from lpm_cases import pkg
from test_gpu_solve_paths import MIXED, System, _body

capi = pkg.capi
pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_records_given_back():
    case = _body(3, (40, 40, 40))
    a = System(case)
    before = _free()
    it = a.solve(MIXED, capi.CG_LOOP_GRAPH)[0]
    takes = before - _free()  # the FP32 operator and vectors
    records = 36 * a.g.nb
    b = System(case)
    K = b.g.K_bsr()
    assert records < takes
    held = torch.empty(_free() - takes + records // 2, dtype=torch.uint8, device="cuda")  # half a set of records short
    try:
        assert b.solve(MIXED, capi.CG_LOOP_GRAPH)[0] == it
        b.g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
        assert np.array_equal(b.g.K_bsr(), K)
    finally:
        del held
        torch.cuda.empty_cache()
    a.g.close()
    b.g.close()
