"""Builds with many atoms per cell in boxes that are large enough for two-cell
tiles: a sample of the list against brute force, from the densities where a tile
of two cells, then of one, no longer fits its shared memory, to those where
none does; and what a build costs there."""
import time

import numpy as np
import pytest

from lammps_b200 import PairLJCut, System

pytestmark = pytest.mark.gpu


def box(per_cell, cells, ntypes, clump=0, s=None):
    """cells^3 cells of the list cutoff 1, per_cell atoms each on the mean."""
    rng = np.random.default_rng(per_cell + cells)
    edge = np.full(3, cells * 1.0001)
    x = rng.random((per_cell * cells**3, 3)) * edge
    if clump:  # one cell with many more
        x[:clump] = 3.0 + 0.9 * rng.random((clump, 3))
    s = s or System("lj", "fp64")
    s.set_box(np.zeros(3), edge)
    p = PairLJCut(0.9, ntypes)
    for t in range(1, ntypes + 1):
        p.coeff(t, t, 1.0, 0.3, 0.9)
    s.set_pair(p)
    s.set_mass([1.0] * ntypes)
    s.set_neighbor(0.1, 1, 0, False)
    s.set_atoms(x, rng.integers(1, ntypes + 1, len(x)).astype(np.int32))
    return s, x, edge


def check_sample(s, x, edge):
    """Every pair that names one of 150 atoms (the first twenty among them)."""
    n = len(x)
    num, jo, ji = s.half_list()
    assert s.neigh_stats()["full_total"] == 2 * len(jo)
    some = np.zeros(n, bool)
    some[::n // 130] = True
    some[:20] = True
    i = np.repeat(np.arange(n), num)
    k = some[i] | some[jo]
    i, jo = i[k].astype(np.int64), jo[k].astype(np.int64)
    got = np.concatenate([(i * n + jo)[some[i]], (jo * n + i)[some[jo]]])
    want = []
    for a in np.nonzero(some)[0]:
        d = x[a] - x
        d -= edge * np.round(d / edge)
        r2 = (d * d).sum(1)
        assert np.abs(r2 - 1.0).min() > 1e-14  # no pair within rounding of the cutoff
        r2[a] = 2.0
        want.append(a * n + np.nonzero(r2 <= 1.0)[0])
    assert np.array_equal(np.sort(got), np.sort(np.concatenate(want)))


@pytest.mark.parametrize("per_cell,cells,ntypes,clump", [
    (52, 11, 1, 0), (110, 11, 1, 0), (145, 11, 2, 0), (170, 11, 1, 0), (40, 11, 1, 600)])
def test_list(per_cell, cells, ntypes, clump):
    s, x, edge = box(per_cell, cells, ntypes, clump)
    s.neigh_build()
    check_sample(s, x, edge)
    s.close()


def seconds(s, builds=10):
    best = 1e9
    for _ in range(builds):
        t = time.perf_counter()
        s.neigh_build()
        best = min(best, time.perf_counter() - t)
    return best


def test_cost_grows_with_the_pairs():
    """A build is bound by its pairs: with four times as many per atom it takes
    about four times as long per atom, and ten times is a path of its own."""
    per_atom = []
    for per_cell in (30, 120):
        s, x, _ = box(per_cell, 12, 1)
        per_atom.append(seconds(s) / len(x))
        s.close()
    assert per_atom[1] < 10 * per_atom[0], per_atom


@pytest.mark.parametrize("clump", [200, 600])  # one tile that needs much memory; one past all
def test_a_clump_costs_no_later_box(clump):
    """The builder's memory per tile follows the current atoms: a box built
    after one with a clump takes the time it takes in a context of its own."""
    s, _, _ = box(20, 20, 1)
    alone = seconds(s)
    box(20, 20, 1, clump, s)
    s.neigh_build()
    s.neigh_build()
    box(20, 20, 1, 0, s)
    s.neigh_build()
    after = seconds(s)
    s.close()
    assert after < 1.5 * alone, (alone, after)  # a third of the resident blocks takes three times


def test_slab():
    """A dense slab in a box three times as long: its mean density is that of a
    thin fluid, its tiles are not.  The list stays the same while the builder
    finds its width and memory, and a build costs what the slab alone costs."""
    s, x, edge = box(125, 11, 1)
    alone = seconds(s)
    s.close()
    s, _, _ = box(125, 11, 1)
    tall = edge * np.array([1.0, 1.0, 3.0])
    s.set_box(np.zeros(3), tall)
    s.set_atoms(x)
    for _ in range(3):
        s.neigh_build()
        check_sample(s, x, tall)
    after = seconds(s)
    s.close()
    assert after < 2.0 * alone, (alone, after)  # ten times by the global-memory path


def test_width_follows_the_box():
    """The width that a slab asked for does not stay for a thin fluid, nor does
    the thin fluid's for the slab."""
    s, x, edge = box(125, 11, 1)
    tall = edge * np.array([1.0, 1.0, 3.0])
    thin, y, wide = box(20, 20, 1)
    alone = seconds(thin)
    thin.close()
    for _ in range(2):
        s.set_box(np.zeros(3), tall)
        s.set_atoms(x)
        for _ in range(3):
            s.neigh_build()
        check_sample(s, x, tall)
        s.set_box(np.zeros(3), wide)
        s.set_atoms(y)
        s.neigh_build()
        check_sample(s, y, wide)
        assert seconds(s) < 1.5 * alone
    s.close()
