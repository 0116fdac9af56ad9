"""Four handles solved at the same time from four host threads, of systems small
enough that their on-chip solves share the SMs: every result is that of the
solve run alone, bit for bit.  One and two slices to a block, in 2-D and 3-D."""
import threading

import numpy as np
import pytest

from lpm_cases import cube, pkg, plate
from test_gpu_two_threads import _handle, _solve

capi = pkg.capi
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,coarse", [(capi.PREC_MIXED, False), (capi.PREC_FP64, False), (capi.PREC_MIXED, True)])
def test_four_threads(precision, coarse):
    jobs = [_handle(c, coarse) for c in (plate(41, 41), plate(61, 121), cube(12), plate(30, 33))]
    alone = [_solve(g, b, precision) for g, b in jobs]
    same = [0] * 4

    def work(k):
        for _ in range(6):
            same[k] += int(np.array_equal(_solve(*jobs[k], precision), alone[k]))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [6] * 4
    assert all(g.onchip_solves() == 7 for g, _ in jobs)
    for g, _ in jobs:
        g.close()
