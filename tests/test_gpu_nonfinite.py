"""An atom whose coordinates have become non-finite takes part in no pair (every
distance test against it is false), as in the reference's pair loops: the
other atoms' forces, energy, virial and steps are bit for bit those of the
same atom moved out of every cutoff, without a new list."""
import os

import numpy as np
import pytest

from lammps_b200 import PairEAM, PairLJCut, System, inputs

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def outcome(style, ntypes, tpa, bad, graphs):
    rng = np.random.default_rng(3)
    eam = style == "eam"
    a = 3.615 if eam else inputs.lj_lattice_constant("fcc", 0.8442)
    x = inputs.lattice("fcc", 6, 6, 6, a)
    hi = np.full(3, 6 * a)
    x = np.mod(x + rng.normal(scale=0.05, size=x.shape), hi)
    n = len(x)
    s = System("metal" if eam else "lj", "fp64")
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
        s.set_mass([1.0] * ntypes)
    s.set_neighbor(1.0 if eam else 0.3, 1000, 0, False)
    s.set_timestep(0.001)
    s.set_thermo(0)
    s.set_launch(tpa)
    s.set_graphs(graphs)
    s.set_atoms(x, rng.integers(1, ntypes + 1, n).astype(np.int32), np.zeros_like(x))
    s.setup()
    moved = x.copy()
    moved[[7, n // 2]] = bad
    s.update_positions(moved)
    r = s.compute(eflag=1, vflag=1)
    f = s.download()["f"]
    row = s.run(9)[-1]
    out = s.download()
    s.close()
    others = np.ones(n, bool)
    others[[7, n // 2]] = False
    return [np.array([r["eng"], *r["virial"], row["E_pair"]]), f[others],
            *(out[k][others] for k in ("x", "v", "f"))]


@pytest.mark.parametrize("style,ntypes", [("lj", 1), ("lj", 3), ("eam", 1)])
@pytest.mark.parametrize("tpa", [1, 4])
@pytest.mark.parametrize("graphs", [True, False])  # many steps a launch, one launch per step
def test_others_unaffected(style, ntypes, tpa, graphs):
    far = outcome(style, ntypes, tpa, [[1.0e6], [2.0e6]], graphs)
    assert all(np.isfinite(u).all() for u in far)
    for bad in (np.nan, np.inf, [3.0, -np.inf, 5.0]):
        for u, v in zip(far, outcome(style, ntypes, tpa, bad, graphs)):
            assert np.array_equal(u, v)
