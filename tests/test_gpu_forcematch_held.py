"""A backward pass uses the list of its forward pass only while the context
still holds those positions."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lammps_b200.forcematch import LJForceField, force_matching_case, pair_matrix  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("between", ["nothing", "other positions", "moved in place", "a build",
                                     "new positions, old list"])
def test_backward_after(between, precision):
    c = force_matching_case(5, 5, 6)
    ff = LJForceField(c["lo"], c["hi"], c["x"], c["types"], 2, 2.9, precision)
    e = pair_matrix(torch.tensor(c["eps"]), 2)
    s = pair_matrix(torch.tensor(c["sigma"]), 2)
    x1 = torch.tensor(c["x"], device="cuda")
    x2 = torch.remainder(x1 + 0.4, torch.tensor(c["hi"], device="cuda")).contiguous()
    g = torch.tensor(np.random.default_rng(1).standard_normal(c["x"].shape), device="cuda")

    def grad(x0, fn=None):
        x = x0.clone().requires_grad_(True)
        f = ff.forces(x, e, s)
        if fn:
            fn(x)
        return torch.autograd.grad((f * g).sum(), x)[0]

    alone, other = grad(x1), grad(x2)
    want = other if between == "moved in place" else alone
    got = grad(x1, {
        "nothing": None,
        "other positions": lambda x: ff.forces(x2, e, s),
        "moved in place": lambda x: x.data.copy_(x2),
        "a build": lambda x: ff.sys.neigh_build(),
        "new positions, old list": lambda x: ff.sys.update_positions(x2.cpu().numpy()),
    }[between])
    ff.close()
    # the same kernel on the same positions and entries; sorting the atoms
    # again after a detour may change the order of FP64 sums
    assert float(torch.linalg.norm(got - want)) <= 1e-12 * float(torch.linalg.norm(want))
