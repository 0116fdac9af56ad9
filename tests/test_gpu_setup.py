"""A lattice's bond arrays and pattern, made on the device from the caller's
list, against a serial restatement: bonds in any order, duplicated bonds,
particles without bonds, a hub with more bonds and candidates than a warp
sorts at once.  Whole numbers: equal; initial lengths: the same operations,
bit for bit."""
import numpy as np
import pytest

from lpm_cases import pkg
from test_gpu_onchip import CASES

capi = pkg.capi
pytestmark = pytest.mark.gpu


def _shuffled(case, seed):
    dim, xyz, p1, p2, layer, Kn, Tv, cell = case
    s = np.random.default_rng(seed).permutation(len(p1))
    return dim, xyz, p1[s], p2[s], layer[s], Kn[s] * (1 + np.arange(len(s))), Tv[s], cell


def _graph(n, pairs, seed):
    """Bonds of the given pairs, both ways, in a random order and layers."""
    rng = np.random.default_rng(seed)
    lay = rng.integers(0, 2, len(pairs))
    p1 = np.concatenate([pairs[:, 0], pairs[:, 1]]).astype(np.int32)
    p2 = np.concatenate([pairs[:, 1], pairs[:, 0]]).astype(np.int32)
    layer = np.concatenate([lay, lay]).astype(np.int32)
    xyz = rng.standard_normal((n, 3))
    case = CASES["cube 3"]()
    return _shuffled((3, xyz, p1, p2, layer, np.ones(len(p1)), np.zeros(len(p1)), case[-1]), seed)


def _hub():
    spokes = np.stack([np.zeros(150, int), np.arange(1, 151)], 1)
    ring = np.stack([np.arange(1, 151), 1 + np.arange(1, 151) % 150], 1)
    return _graph(151, np.concatenate([spokes, ring]), 3)


SETUPS = {
    "cube 3 shuffled": lambda: _shuffled(CASES["cube 3"](), 1),
    "plate 13x29 shuffled": lambda: _shuffled(CASES["plate 13x29"](), 2),
    "cube renumbered": lambda: CASES["cube renumbered"](),
    "hub": _hub,                                                     # 150 bonds, up to 23k candidates
    "one pair": lambda: _graph(2, np.array([[0, 1]]), 4),
    "some without bonds": lambda: _graph(40, np.array([[3, 9], [9, 11], [11, 3], [30, 31]]), 5),
    "a pair twice": lambda: _graph(5, np.array([[0, 1], [0, 1], [0, 1], [1, 2], [2, 3]]), 6),
}


@pytest.mark.parametrize("name", list(SETUPS))
def test_setup_matches_a_serial_pass(name):
    dim, xyz, p1, p2, layer, Kn, Tv, cell = SETUPS[name]()
    n = len(xyz)
    g = capi.Lattice(dim, xyz, p1, p2, layer, Kn, Tv, cell.particle_volume, cell.nneighbors)
    got = g.bonds()
    order = np.lexsort((layer, p1))
    assert np.array_equal(g.bond_perm, order)
    q1, q2, ql = p1[order], p2[order], layer[order]
    assert np.array_equal(got["bp2"], q2) and np.array_equal(got["blayer"], ql)
    assert np.array_equal(got["bptr"], np.searchsorted(q1, np.arange(n + 1)))
    assert np.array_equal(g.download(capi.B_KN), Kn[order])
    dx = xyz[q1] - xyz[q2]
    assert np.array_equal(g.download(capi.B_DIS0), np.sqrt(dx[:, 0] * dx[:, 0] + dx[:, 1] * dx[:, 1] + dx[:, 2] * dx[:, 2]))
    first = {}
    for b, k in enumerate(zip(q1.tolist(), q2.tolist(), ql.tolist())):
        first.setdefault(k, b)
    assert np.array_equal(got["opp"], [first[k] for k in zip(q2.tolist(), q1.tolist(), ql.tolist())])
    nbrs = [[q2[(q1 == i) & (ql == l)] for l in (0, 1)] for i in range(n)]
    cptr, cidx = g.pattern()
    for i in range(n):
        c = [np.concatenate([[k], nbrs[k][l]]) for l in (0, 1) for k in nbrs[i][l]]
        assert np.array_equal(cidx[cptr[i]:cptr[i + 1]], np.unique(np.concatenate(c)) if c else [])
    g.close()


def test_setup_refuses_a_bond_without_its_opposite():
    dim, xyz, p1, p2, layer, Kn, Tv, cell = CASES["cube 3"]()
    keep = np.arange(len(p1)) != 7
    with pytest.raises(capi.LpmError, match="opposite"):
        capi.Lattice(dim, xyz, p1[keep], p2[keep], layer[keep], Kn[keep], Tv[keep], cell.particle_volume, cell.nneighbors)
    other = layer.copy()
    other[7] = 1 - other[7]
    with pytest.raises(capi.LpmError, match="opposite"):
        capi.Lattice(dim, xyz, p1, p2, other, Kn, Tv, cell.particle_volume, cell.nneighbors)
