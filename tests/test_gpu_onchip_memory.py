"""A solve past the on-chip limits takes no memory for a plan that it cannot
use: on a handle whose other solve has run, the device's free memory is the
same before and after."""
import pytest
import torch

from lpm_cases import pkg
from test_gpu_solve_paths import FP64, MIXED, System, _body

capi = pkg.capi
pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("dim,size,precision", [(2, (250, 245), FP64), (3, (40, 40, 40), FP64), (3, (43, 43, 43), MIXED)])
def test_refused_solve_takes_no_memory(dim, size, precision):
    warm = System(_body(dim, size))  # the kernels' own memory, loaded with their first launch
    warm.solve(precision, capi.CG_LOOP_GRAPH)
    warm.solve(precision, capi.CG_LOOP_PERSISTENT)
    s = System(_body(dim, size))
    s.solve(precision, capi.CG_LOOP_GRAPH)
    before = _free()
    assert s.solve(precision, capi.CG_LOOP_PERSISTENT)[1:] == (1, 0)
    assert _free() == before
    warm.g.close()
    s.g.close()
