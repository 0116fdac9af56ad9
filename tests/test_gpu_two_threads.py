"""Two handles solved at the same time from two host threads: each on-chip
solve (one cooperative launch that fills the GPU) takes its turn, and every
result is that of the solve run alone, bit for bit."""
import threading

import numpy as np
import pytest

from lpm_cases import cube, make_gpu, pkg, plate
from test_gpu_onchip import TOL

capi = pkg.capi
pytestmark = pytest.mark.gpu


def _handle(case, coarse):
    dim, xyz = case[0], case[1]
    g = make_gpu(*case)
    mask = np.zeros((g.n, 3), np.int32)
    mask[xyz[:, dim - 1] < xyz[:, dim - 1].min() + 1e-9, :dim] = 1
    g.set_mask(mask)
    if coarse:
        g.set_preconditioner(capi.PRECOND_COARSE, 0.0)
    g.update()
    g.assemble(capi.TANGENT_SYMMETRIC, capi.BC_ELIMINATE)
    b = (np.random.default_rng(g.n).standard_normal((g.n, dim)) * (1 - mask[:, :dim])).ravel()
    return g, b


def _solve(g, b, precision):
    g.upload(capi.F_RESIDUAL, b)
    assert g.solve(precision, TOL)[2] == capi.OK
    return g.download(capi.F_DISP)


@pytest.mark.parametrize("precision,coarse", [(capi.PREC_MIXED, False), (capi.PREC_FP64, False), (capi.PREC_MIXED, True)])
def test_two_threads(precision, coarse):
    jobs = [_handle(plate(60, 61), coarse), _handle(cube(14), coarse)]
    alone = [_solve(g, b, precision) for g, b in jobs]
    same = [0, 0]

    def work(k):
        for _ in range(8):
            same[k] += int(np.array_equal(_solve(*jobs[k], precision), alone[k]))

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert same == [8, 8]
    for g, _ in jobs:
        g.close()
