"""Launches of several MD steps against one launch per step: the same run must
end in the same bits (positions, velocities, forces, image flags, thermo rows,
build counts), at every launch shape and list schedule, through rebuilds and
output steps.  With graphs off the engine steps one launch at a time."""
import os

import numpy as np
import pytest

from lammps_b200 import PairEAM, PairLJCut, System, inputs

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def run(single, style, precision, tpa, cells, drop, ntypes, schedule, steps, thermo):
    rng = np.random.default_rng(sum(cells) + drop)
    eam = style == "eam"
    a = 3.615 if eam else inputs.lj_lattice_constant("fcc", 0.8442)
    x = inputs.lattice("fcc", *cells, a)
    hi = np.array(cells) * a
    x = np.mod(x + rng.normal(scale=0.05, size=x.shape), hi)[drop:]
    n = len(x)
    s = System("metal" if eam else "lj", precision)
    s.set_box(np.zeros(3), hi)
    if eam:
        p = PairEAM(1)
        p.coeff(1, os.path.join(GOLDEN, "Cu_u3.eam"))
        s.set_pair(p)
    else:
        p = PairLJCut(2.5, ntypes)
        for t in range(1, ntypes + 1):
            p.coeff(t, t, 1.0, 1.0 - 0.03 * t, 2.5)
        s.set_pair(p)
        s.set_mass([1.0 + t for t in range(ntypes)])
    every, delay, check = schedule
    s.set_neighbor(1.0 if eam else 0.3, every, delay, check)
    s.set_timestep(0.005)
    s.set_thermo(thermo)
    s.set_launch(tpa)
    if single:
        s.set_graphs(False)
    v = rng.normal(scale=4.0 if eam else 1.2, size=x.shape)
    s.set_atoms(x, rng.integers(1, ntypes + 1, n).astype(np.int32), v - v.mean(0))
    s.setup()
    l0 = s.kernel_launches
    rows = s.run(steps) + s.run(7)  # a second run starts from the first one's state
    out = s.download()
    out["rows"] = np.array([[r["Step"], r["Temp"], r["E_pair"], r["Press"]] for r in rows])
    st = s.neigh_stats()
    launches = s.kernel_launches - l0
    s.close()
    return out, (st["ncalls"], st["ndanger"], st["full_total"]), launches


CASES = [
    # style, types, cells, sites left out, (every, delay, check), steps, thermo
    ("lj", 1, (5, 5, 5), 1, (20, 0, False), 61, 0),
    ("lj", 1, (6, 6, 6), 0, (1, 3, True), 60, 25),
    ("lj", 3, (8, 8, 8), 3, (5, 0, True), 47, 10),
    ("lj", 1, (12, 12, 12), 0, (7, 0, False), 40, 0),
    ("eam", 1, (5, 6, 5), 1, (1, 5, True), 45, 20),
    ("eam", 1, (10, 10, 10), 0, (10, 0, False), 33, 0),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tpa", [1, 2, 4, 8])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-{c[2][0]}")
def test_same_bits_as_one_launch_per_step(case, tpa, precision):
    style, ntypes, cells, drop, schedule, steps, thermo = case
    many, nb, lm = run(False, style, precision, tpa, cells, drop, ntypes, schedule, steps, thermo)
    one, nb1, l1 = run(True, style, precision, tpa, cells, drop, ntypes, schedule, steps, thermo)
    assert nb == nb1
    assert lm < l1  # the runs took different forms
    for k in ("x", "v", "f", "image", "rows"):
        assert np.array_equal(many[k], one[k]), k


def test_long_chunks():
    """A chunk of 256 steps in one launch, then the rest of the run."""
    args = ("lj", "mixed", 8, (5, 5, 5), 0, 1, (1000, 0, False), 300, 0)
    many, _, _ = run(False, *args)
    one, _, _ = run(True, *args)
    for k in ("x", "v", "f", "image", "rows"):
        assert np.array_equal(many[k], one[k]), k
