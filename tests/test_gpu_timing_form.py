"""Timing mode 2 keeps the form that the run takes without timers: the same
launches and bits, also where several steps run in one launch, with every
step's time accounted for."""
import numpy as np
import pytest

from lammps_b200 import PairLJCut, System, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [6, 20])
@pytest.mark.parametrize("schedule", [(20, 0, False), (1, 3, True)])
def test_same_form(cells, schedule):
    rng = np.random.default_rng(cells)
    a = inputs.lj_lattice_constant("fcc", 0.8442)
    x = np.mod(inputs.lattice("fcc", cells, cells, cells, a) + rng.normal(scale=0.05, size=(
        4 * cells**3, 3)), cells * a)
    v = rng.normal(size=x.shape)
    out = []
    for mode in (0, 2):
        s = System("lj", "mixed")
        s.set_box([0.0] * 3, [cells * a] * 3)
        p = PairLJCut(2.5)
        p.coeff(1, 1, 1.0, 1.0, 2.5)
        s.set_pair(p)
        s.set_mass([1.0])
        s.set_neighbor(0.3, *schedule)
        s.set_timestep(0.004)
        s.set_thermo(50)
        s.set_launch(4)
        s.set_atoms(x, None, v)
        s.setup()
        s.set_timing(mode)
        l0 = s.kernel_launches
        s.run(300)
        out.append([s.download()["x"], s.kernel_launches - l0])
        if mode:
            t = s.timing()
            ms = s.step_times()
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
    assert t["steps"] == len(ms) == 300
    total = t["initial"] + t["neigh"] + t["pair1"]
    assert t["pair2"] == t["final"] == 0.0 and (np.asarray(ms) > 0).all()
    assert abs(np.sum(ms) - total) <= 1e-4 * total  # FP32 times
