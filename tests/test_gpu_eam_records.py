"""The position and F' records of one-element eam: memory that only such a
context holds, there whichever of style and atoms comes first and however the
atom count changes."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lammps_b200 import PairEAM, PairLJCut, System, inputs  # noqa: E402

pytestmark = pytest.mark.gpu
CU = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "Cu_u3.eam")


def eam():
    p = PairEAM(1)
    p.coeff(1, CU)
    return p


def test_memory_of_other_styles():
    n, used = 1_000_000, {}
    x = np.random.default_rng(0).random((n, 3)) * 300.0
    lj = PairLJCut(2.5)
    lj.coeff(1, 1, 1.0, 1.0, 2.5)
    for style, pair in (("lj", lj), ("metal", eam())):
        s = System(style, "fp64")
        s.set_box([0.0] * 3, [300.0] * 3)
        s.set_pair(pair)
        if style == "lj":
            s.set_mass([1.0])
        before = torch.cuda.mem_get_info()[0]
        s.set_atoms(x)
        used[style] = before - torch.cuda.mem_get_info()[0]
        s.close()
    # 32 bytes an atom, less what the allocator's 2 MB blocks round away
    assert used["metal"] - used["lj"] > 32 * n - (4 << 20), used


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_either_order(precision):
    rng = np.random.default_rng(1)

    def forces(s, cells):
        x = inputs.lattice("fcc", *cells, 3.615) + 0.02 * rng.standard_normal((4 * np.prod(cells), 3))
        s.set_box([0.0] * 3, np.array(cells) * 3.615)
        s.set_atoms(x)
        return x

    def compute(s):
        s.neigh_build()
        r = s.compute(eflag=1, vflag=1)
        return [s.download()["f"], r["eng"], r["virial"]]

    late = System("metal", precision)
    late.set_mass([63.55])
    late.set_neighbor(1.0, 1, 0, False)
    late.set_launch(2)
    for k, cells in enumerate([(6, 6, 6), (5, 5, 5), (9, 9, 9)]):
        x = forces(late, cells)
        if k == 0:
            late.set_pair(eam())  # after the atoms
        got = compute(late)
        s = System("metal", precision)
        s.set_pair(eam())
        s.set_neighbor(1.0, 1, 0, False)
        s.set_launch(2)
        s.set_box([0.0] * 3, np.array(cells) * 3.615)
        s.set_atoms(x)
        for u, v in zip(got, compute(s)):
            assert np.array_equal(u, v)
        s.close()
    late.close()
