"""Launches of several MD steps in the kernels that the other multi-step tests
do not reach, against one launch per step, bit for bit: eam with two elements
(symmetric and unsymmetric densities), boxes with three and four blocks per SM,
and a list that outgrows its capacity in the middle of such a run."""
import os

import numpy as np
import pytest

from lammps_b200 import PairEAM, PairEAMAlloy, PairEAMFS, PairLJCut, System, inputs
from test_gpu_eam_multi import write_two_element

pytestmark = pytest.mark.gpu
CU = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "Cu_u3.eam")


def pair_of(style, tmp_path):
    if style in ("alloy", "fs"):
        p = (PairEAMFS if style == "fs" else PairEAMAlloy)(2)
        p.coeff(write_two_element(str(tmp_path / f"ab.eam.{style}"), style == "fs"), ["A", "B"])
        return p, 2, 3.6
    if style == "eam":
        p = PairEAM(1)
        p.coeff(1, CU)
        return p, 1, 3.615
    nt = int(style[2:])
    p = PairLJCut(2.5, nt)
    for t in range(1, nt + 1):
        p.coeff(t, t, 1.0, 1.0 - 0.03 * t, 2.5)
    return p, nt, inputs.lj_lattice_constant("fcc", 0.8442)


def both_forms(style, precision, tpa, cells, schedule, steps, tmp_path, **kw):
    out = []
    for graphs in (True, False):
        pair, nt, a = pair_of(style, tmp_path)
        rng = np.random.default_rng(cells + nt)
        lj = style.startswith("lj")
        x = kw["x"] if "x" in kw else np.mod(inputs.lattice("fcc", cells, cells, cells, a) +
                                             rng.normal(scale=0.05, size=(4 * cells**3, 3)), cells * a)
        edge = kw.get("edge", cells * a)
        s = System("lj" if lj else "metal", precision)
        s.set_box([0.0] * 3, [edge] * 3)
        if "cut" in kw:
            pair = PairLJCut(kw["cut"])
            pair.coeff(1, 1, 1.0, 0.8, kw["cut"])
        s.set_pair(pair)
        if lj:
            s.set_mass([1.0] * nt)
        s.set_neighbor(kw.get("skin", 0.3 if lj else 1.0), *schedule, kw.get("one", 0))
        s.set_timestep(kw.get("dt", 0.004 if lj else 0.002))
        s.set_thermo(15)
        s.set_launch(tpa)
        s.set_graphs(graphs)
        v = rng.normal(scale=1.2 if lj else 4.0, size=x.shape)
        s.set_atoms(x, rng.integers(1, nt + 1, len(x)).astype(np.int32), v - v.mean(0))
        s.setup()
        cap = s.neigh_stats()["capacity"]
        l0 = s.kernel_launches
        rows = s.run(steps)
        launches = s.kernel_launches - l0
        o = s.download()
        o["rows"] = np.array([[r["Step"], r["Temp"], r["E_pair"], r["Press"]] for r in rows])
        st = s.neigh_stats()
        s.close()
        out.append((o, (st["ncalls"], st["ndanger"], st["full_total"]), launches, cap, st["capacity"]))
    many, one = out
    assert many[2] < one[2]  # the runs took different forms
    assert many[1] == one[1]
    for k in ("x", "v", "f", "image", "rows"):
        assert np.array_equal(many[0][k], one[0][k]), k
    return many


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tpa", [1, 2, 4, 8])
@pytest.mark.parametrize("style", ["alloy", "fs"])
def test_two_elements(style, tpa, precision, tmp_path):
    both_forms(style, precision, tpa, 6, (1, 3, True), 47, tmp_path)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
# threads over 256 a block and the SMs: 14^3 x 8 and 20^3 x 4 give three and four
@pytest.mark.parametrize("cells,tpa", [(14, 8), (20, 4), (25, 2)])
@pytest.mark.parametrize("style", ["lj1", "lj3", "eam", "alloy"])
def test_full_chip(style, cells, tpa, precision, tmp_path):
    both_forms(style, precision, tpa, cells, (10, 0, False), 33, tmp_path)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_overflow_in_mid_chunk(precision, tmp_path):
    # six neighbours an atom on the lattice, room for eight, more when it melts
    m = 12
    g = np.arange(m) * 1.25 + 0.3
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    r = both_forms("lj1", precision, 2, 0, (5, 0, False), 200, tmp_path, x=x, edge=m * 1.25,
                   cut=1.2, skin=0.2, one=-8, dt=0.003)
    assert r[3] == 8 and r[4] > 8


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_long_chunk(precision, tmp_path):
    """More than the 256 steps of a chunk without a rebuild."""
    both_forms("lj1", precision, 8, 5, (1000, 0, False), 300, tmp_path, dt=0.0005, skin=0.8)
