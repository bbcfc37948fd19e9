"""The order of a list's entries, which fixes the order of every FP64 sum: by
neighbour cell (z slowest, x fastest) and inside a cell by caller index, for
the one-launch sort, the sort of larger boxes and both widths of tile."""
import numpy as np
import pytest

from lammps_b200 import PairLJCut, System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,edge,cut", [
    (900, (5.0, 5.6, 6.1), 1.0),      # a few cells, one-cell tiles
    (8000, (14.0, 15.0, 13.5), 1.0),  # two-cell tiles, one-launch sort
    (300, (3.1, 3.4, 3.3), 1.6),      # one and two cells per edge
    (3000, (28.0, 28.0, 26.0), 0.9),  # more cells than the one-launch sort takes
    (160000, (38.0, 41.0, 39.0), 1.0),  # more atoms than it takes
])
def test_order(n, edge, cut):
    rng = np.random.default_rng(n)
    edge = np.array(edge)
    x = rng.random((n, 3)) * edge
    s = System("lj", "fp64")
    s.set_box(np.zeros(3), edge)
    p = PairLJCut(cut)
    p.coeff(1, 1, 1.0, 0.3, cut)
    s.set_pair(p)
    s.set_mass([1.0])
    s.set_neighbor(0.1, 1, 0, False)
    s.set_atoms(x)
    s.neigh_build()
    num, j, image = s.half_list()
    s.close()
    nc = np.maximum((edge / (cut + 0.1)).astype(int), 1)
    cell = np.minimum((x * (nc / edge)).astype(int), nc - 1)
    i = np.repeat(np.arange(n), num)
    shift = np.stack([image % 3, image // 3 % 3, image // 9], 1) - 1
    d = cell[j] + shift * nc - cell[i]
    assert (np.abs(d) <= 1).all()
    key = (((d[:, 2] + 1) * 3 + d[:, 1] + 1) * 3 + d[:, 0] + 1) * np.int64(n) + j
    same = i[1:] == i[:-1]
    assert same.sum() > 100  # neighbours compared (few in the dilute box)
    assert (np.diff(key)[same] > 0).all()
