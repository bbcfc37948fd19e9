"""The cell sort of a list build at the edges of its blocks and cells: wrapped
positions and image flags against the same arithmetic in numpy, every atom
kept exactly once, and repeated builds that change nothing."""
import numpy as np
import pytest

from lammps_b200 import PairLJCut, System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
# (atoms, edges): one cell, exactly filled blocks, one over, cells at and past
# the most that one block scans (16,383), atoms past the one-launch sort
@pytest.mark.parametrize("n,edge", [(1, (3.0, 3.0, 3.0)), (255, (7.0, 7.0, 7.0)),
                                    (256, (7.0, 8.0, 9.0)), (257, (2.9, 30.0, 2.9)),
                                    (5000, (26.0, 26.0, 26.0)), (3000, (28.0, 28.0, 26.0)),
                                    (160000, (40.0, 41.0, 39.0))])
def test_sort(n, edge, precision):
    rng = np.random.default_rng(n)
    edge = np.array(edge)
    lo = np.array([-3.0, 0.0, 11.0])
    x = lo + rng.uniform(-0.9, 1.9, (n, 3)) * edge  # up to one box outside
    v = rng.standard_normal((n, 3))
    s = System("lj", precision)
    s.set_box(lo, lo + edge)
    p = PairLJCut(0.9)
    p.coeff(1, 1, 1.0, 1.0, 0.9)
    s.set_pair(p)
    s.set_mass([1.0])
    s.set_neighbor(0.1, every=1, delay=0, check=True)
    s.set_atoms(x, None, v)
    s.neigh_build()
    one = s.download()
    want, image = x.copy(), np.zeros((n, 3), np.int32)
    under = want < lo
    want = np.where(under, want + edge, want)
    over = want >= lo + edge
    want = np.where(over, np.maximum(want - edge, lo), want)
    image = image - under.astype(np.int32) + over.astype(np.int32)
    assert np.array_equal(one["x"], want)
    assert np.array_equal(one["image"], image)
    assert np.array_equal(one["v"], v)
    total = s.neigh_stats()["full_total"]
    s.neigh_build()
    two = s.download()
    for k in ("x", "v", "image"):
        assert np.array_equal(one[k], two[k])
    assert s.neigh_stats()["full_total"] == total
    s.close()
