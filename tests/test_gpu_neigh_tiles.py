"""The tiled list builder against brute force, at the sizes where its tiles,
chunks and acceptance band can go wrong: the list must equal the FP64
criterion exactly (whole sets and counts, no tolerance)."""
import numpy as np
import pytest

from lammps_b200 import PairLJCut, System

pytestmark = pytest.mark.gpu


def brute(x, types, edge, cutsq):
    """Directed pairs (i, j, image code) with the reference's arithmetic."""
    out = []
    cut = np.sqrt(cutsq.max())
    for s in np.ndindex(3, 3, 3):
        s = np.array(s) - 1
        near = np.ones(len(x), bool)
        for d in range(3):  # image atoms that can reach the box
            if s[d] < 0:
                near &= x[:, d] - edge[d] >= x[:, d].min() - cut - 1e-6
            elif s[d] > 0:
                near &= x[:, d] + edge[d] <= x[:, d].max() + cut + 1e-6
        j = np.nonzero(near)[0]
        if len(j) == 0:
            continue
        xj = x[j] + s * edge
        for a in range(0, len(x), 512):
            d = x[a:a + 512, None, :] - xj[None]
            r2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
            hit = r2 <= cutsq[types[a:a + 512, None], types[None, j]]
            i, k = np.nonzero(hit)
            i = i + a
            if not s.any():
                keep = i != j[k]
                i, k = i[keep], k[keep]
            code = (s[0] + 1) + 3 * (s[1] + 1) + 9 * (s[2] + 1)
            out.append(np.stack([i, j[k], np.full(len(i), code)], 1))
    return np.concatenate(out).astype(np.int64)


def keys(p, n):
    return np.sort((p[:, 0] * n + p[:, 1]) * 27 + p[:, 2])


def check(x, types, lo, edge, cuts, skin):
    nt = len(cuts)
    s = System("lj", "fp64")
    s.set_box(lo, lo + edge)
    p = PairLJCut(max(cuts), nt)
    for a in range(nt):
        for b in range(a, nt):
            p.coeff(a + 1, b + 1, 1.0, 1.0, np.sqrt(cuts[a] * cuts[b]))
    s.set_pair(p)
    s.set_mass([1.0] * nt)
    s.set_neighbor(skin, every=1, delay=0, check=False)
    s.set_atoms(x, types)
    s.neigh_build()
    n = len(x)
    t = s.tables["cutsq"].reshape(nt + 1, nt + 1)
    cutsq = (np.sqrt(t) + skin) ** 2
    ref = brute(x, types, edge, cutsq)
    num, jo, ji = s.half_list()
    half = np.stack([np.repeat(np.arange(n), num), jo, ji], 1).astype(np.int64)
    back = np.stack([half[:, 1], half[:, 0], 26 - half[:, 2]], 1)
    got = keys(np.concatenate([half, back]), n)
    assert s.neigh_stats()["full_total"] == len(ref)
    assert np.array_equal(got, keys(ref, n))
    s.close()


CASES = {
    # name: (atoms, edges, cutoffs per type, skin, lo)
    "few atoms, empty cells": (700, (30.0, 28.0, 31.0), [0.9], 0.1, 0.0),
    "two cells per edge": (500, (2.3, 2.4, 2.2), [0.8], 0.2, 0.0),
    "one cell per edge": (180, (1.5, 1.7, 1.9), [0.8], 0.2, 0.0),
    "one cell, too many chunks to stage": (330, (1.5, 1.7, 1.9), [0.8], 0.2, 0.0),
    "fifty atoms per cell": (1500, (3.7, 3.8, 3.9), [1.0], 0.2, 0.0),
    "odd row of two-cell tiles": (3000, (13.3, 9.2, 9.1), [0.9], 0.1, 0.0),
    "wide flat cells": (400, (5000.0, 6.0, 6.0), [0.9], 0.1, 0.0),
    "far from the origin": (900, (6.0, 7.0, 5.5), [1.0], 0.3, -4.0e4),
    "large units": (900, (1800.0, 2100.0, 1650.0), [300.0], 90.0, 0.0),
    "small units": (900, (6e-3, 7e-3, 5.5e-3), [1e-3], 3e-4, 0.0),
    "three types": (1200, (9.0, 8.0, 10.0), [1.0, 1.6, 2.2], 0.25, 0.0),
    "eight types": (1200, (9.0, 8.0, 10.0), [1.0, 1.1, 1.2, 1.3, 1.5, 1.7, 2.0, 2.2], 0.25, 0.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_list_equals_brute_force(name):
    n, edge, cuts, skin, lo = CASES[name]
    rng = np.random.default_rng(len(name))
    edge = np.array(edge)
    lo = np.full(3, lo)
    x = np.minimum(lo + rng.random((n, 3)) * edge, np.nextafter(lo + edge, lo))
    types = rng.integers(1, len(cuts) + 1, n).astype(np.int32)
    check(x, types, lo, edge, cuts, skin)


@pytest.mark.parametrize("shift", [0.0, 0.125])
def test_pairs_exactly_at_the_cutoff(shift):
    # spacing 0.5, list cutoff 1.5: whole shells sit exactly on the cutoff
    g = np.arange(12) * 0.5 + shift
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    check(x, np.ones(len(x), np.int32), np.zeros(3), np.full(3, 6.0), [1.25], 0.25)


def test_pairs_around_the_cutoff():
    # 1,000 pairs of separations within 1e-9 .. 1e-4 of the list cutoff
    rng = np.random.default_rng(5)
    n = 1000
    a = rng.random((n, 3)) * 60.0
    u = rng.standard_normal((n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    off = 10.0 ** rng.uniform(-9, -4, n) * rng.choice([-1.0, 1.0], n)
    b = np.mod(a + u * (1.3 + off)[:, None], 60.0)
    x = np.concatenate([a, b])
    check(x, np.ones(2 * n, np.int32), np.zeros(3), np.full(3, 60.0), [1.0], 0.3)
