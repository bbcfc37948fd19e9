"""A grid barrier that gives up (here: at once, by b200_expire_waits) is an
error of the call, not of the context: nothing of the abandoned launch is left
for the next one, and the same atoms uploaded again give the bits of a fresh
context."""
import numpy as np
import pytest

from lammps_b200 import PairLJCut, System, inputs
from lammps_b200._abi import B200Error
from lammps_b200.replicas import make_batch, replica_batch

pytestmark = pytest.mark.gpu
TIMEOUT, STATE = -8, -4


def expire(s, on):
    s._ck(s._L.b200_expire_waits(s._h, on))


def gives_up(call):
    with pytest.raises(B200Error) as e:
        call()
    assert e.value.code == TIMEOUT
    assert "timed out" in str(e.value)


def no_atoms(call):
    with pytest.raises(B200Error) as e:
        call()
    assert e.value.code == STATE


class Box:
    def __init__(self, precision, check=False, tpa=2, cells=9, spread=1.0):
        rng = np.random.default_rng(cells)
        a = inputs.lj_lattice_constant("fcc", 0.8442) * spread
        x = inputs.lattice("fcc", cells, cells, cells, a)
        self.hi = np.full(3, cells * a)
        self.x = np.mod(x + rng.normal(scale=0.04, size=x.shape), self.hi)
        self.v = rng.normal(size=x.shape)
        self.precision, self.check, self.tpa = precision, check, tpa
        self.cut = 2.5 if spread == 1.0 else 0.9

    def system(self):
        s = System("lj", self.precision)
        s.set_box(np.zeros(3), self.hi)
        p = PairLJCut(self.cut)
        p.coeff(1, 1, 1.0, 1.0 if self.cut == 2.5 else 0.5, self.cut)
        s.set_pair(p)
        s.set_mass([1.0])
        s.set_neighbor(0.3 if self.cut == 2.5 else 0.1, 5, 0, self.check)
        s.set_launch(self.tpa)
        return s

    def result(self, s, steps):
        s.set_atoms(self.x, None, self.v)
        if steps:
            s.setup()
            s.run(steps)
        else:
            s.neigh_build()
            s.compute()
        out = s.download()
        st = s.neigh_stats()
        return [out["x"], out["v"], out["f"], st["full_total"]]


def same(a, b):
    assert all(np.array_equal(u, v) for u, v in zip(a, b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sort(precision):
    b = Box(precision)
    s, t = b.system(), b.system()
    s.set_atoms(b.x, None, b.v)
    expire(s, 1)
    gives_up(s.neigh_build)  # the first build: no cell start was ever written
    for call in (s.neigh_build, s.compute, s.download):
        no_atoms(call)
    for _ in range(3):
        s.set_atoms(b.x, None, b.v)
        gives_up(s.neigh_build)
    expire(s, 0)
    same(b.result(s, 0), b.result(t, 0))
    s.close()
    t.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("check", [False, True])
def test_steps(precision, check):
    b = Box(precision, check)
    s, t = b.system(), b.system()
    s.set_atoms(b.x, None, b.v)
    s.setup()
    s.run(12)
    expire(s, 1)
    gives_up(lambda: s.run(30))
    for call in (s.compute, s.download, lambda: s.run(5)):
        no_atoms(call)
    expire(s, 0)
    same(b.result(s, 40), b.result(t, 40))
    s.close()
    t.close()


def test_launch_shape_search():
    # more cells than the one-launch sort takes: only the search's own
    # launches of several steps wait
    b = Box("mixed", tpa=0, cells=9, spread=1.9)
    s = b.system()
    s.set_atoms(b.x, None, b.v)
    expire(s, 1)
    gives_up(s.setup)
    expire(s, 0)
    s.set_atoms(b.x, None, b.v)
    s.setup()
    s.run(20)
    assert np.isfinite(s.download()["x"]).all()
    s.close()


def test_replica_batch():
    batch = replica_batch(nrep=6, seed=12345)
    s, t = make_batch(batch, "mixed", tpa=1), make_batch(batch, "mixed", tpa=1)
    expire(s, 1)
    gives_up(s.neigh_build)
    expire(s, 0)
    out = []
    for q in (s, t):
        q.set_atoms(batch["x"], batch.get("types"), batch["v"])
        q.neigh_build()
        q.compute()
        out.append([q.download()["f"], q.neigh_stats()["full_total"]])
        q.close()
    same(*out)
