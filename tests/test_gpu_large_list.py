"""A list of more particles than 2^20 blocks of the pattern's four (a warp
each): the bonds are among the last ones, and their rows of the pattern are
those of a chain."""
import numpy as np
import pytest

from lpm_cases import pkg

capi = pkg.capi
pytestmark = pytest.mark.gpu


def test_pattern_of_the_last_particles():
    n, m = 4 * 2**20 + 1000, 500
    i = np.arange(n - m, n - 1)
    p1 = np.concatenate([i, i + 1]).astype(np.int32)
    p2 = np.concatenate([i + 1, i]).astype(np.int32)
    xyz = np.zeros((n, 3))
    xyz[:, 0] = np.arange(n)
    g = capi.Lattice(2, xyz, p1, p2, np.zeros(len(p1), np.int32), np.ones(len(p1)), np.zeros(len(p1)), 1.0, 2)
    cptr, cidx = g.pattern()
    g.close()
    assert not cptr[:n - m + 1].any()
    for k in range(n - m, n):  # the partners and their partners, itself among them
        row = [j for j in range(k - 2, k + 3) if n - m <= j < n]
        assert cidx[cptr[k]:cptr[k + 1]].tolist() == row
