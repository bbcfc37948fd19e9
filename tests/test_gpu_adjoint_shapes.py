"""Force-matching forward and backward at every threads-per-atom shape and
number of types, against plain torch in FP64 over a k-d tree's pairs.

Tolerances, norm-wise relative: FP64 sums of about a hundred rounded terms
whose size is up to a thousand times the result's, 1e-11; mixed, FP32 pair
arithmetic, the engine's 1e-5 bar.  The mixed form decides the cutoff in FP32:
the force jumps there, so the atoms of pairs within 1e-6 (relative, of r^2) of
it are left out of the per-atom comparisons."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from lammps_b200 import inputs  # noqa: E402
from lammps_b200.forcematch import LJForceField, pair_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
CUT = 2.5


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("cells,ntypes,drop", [((6, 6, 7), 3, 1), ((14, 14, 14), 1, 0),
                                               ((16, 16, 17), 4, 3), ((20, 20, 21), 2, 5)])
def test_forward_backward(cells, ntypes, drop, precision, tol):
    from scipy.spatial import cKDTree

    rng = np.random.default_rng(sum(cells) + ntypes)
    a = inputs.lj_lattice_constant("fcc", 0.85)
    x = inputs.lattice("fcc", *cells, a)
    hi = np.array(cells) * a
    x = np.mod(x + rng.normal(scale=0.05, size=x.shape), hi)[drop:]
    n = len(x)
    t = rng.integers(1, ntypes + 1, n).astype(np.int32)
    m = ntypes * (ntypes + 1) // 2
    eps = torch.tensor(rng.uniform(0.5, 1.5, m), requires_grad=True)
    sig = torch.tensor(rng.uniform(0.92, 1.08, m), requires_grad=True)
    g = torch.tensor(rng.standard_normal((n, 3)))

    ff = LJForceField(np.zeros(3), hi, x, t, ntypes, CUT * 1.08, precision)
    xd = torch.tensor(x, device="cuda").requires_grad_(True)
    f = ff.forces(xd, pair_matrix(eps, ntypes), pair_matrix(sig, ntypes), cut_factor=CUT)
    got = torch.autograd.grad((f * g.cuda()).sum(), (xd, eps, sig))
    ff.close()

    p = cKDTree(x, boxsize=hi).query_pairs(CUT * 1.08, output_type="ndarray")
    i, j = (torch.tensor(np.concatenate([p[:, k], p[:, 1 - k]])) for k in (0, 1))
    xr = torch.tensor(x, requires_grad=True)
    L = torch.tensor(hi)
    d = xr[i] - xr[j]
    d = d - L * torch.round((d / L).detach())
    r2 = (d * d).sum(1)
    tt = (torch.tensor(t).long()[i], torch.tensor(t).long()[j])
    e, s = pair_matrix(eps, ntypes)[tt], pair_matrix(sig, ntypes)[tt]
    r6 = 1.0 / r2**3
    w = (48 * e * s**12 * r6 - 24 * e * s**6) * r6 / r2
    w = torch.where(r2 < (CUT * s.detach()) ** 2, w, torch.zeros_like(w))
    fr = torch.zeros_like(xr).index_add(0, i, d * w[:, None])
    ref = torch.autograd.grad((fr * g).sum(), (xr, eps, sig))

    keep = torch.ones(n, dtype=torch.bool)
    if precision == "mixed":
        edge = (r2 / (CUT * s) ** 2 - 1).abs() < 1e-6
        keep[i[edge]] = False
    assert keep.sum() > 0.99 * n

    def rel(u, v):
        u, v = u.detach().cpu(), v.detach()
        if len(u) == n:
            u, v = u[keep], v[keep]
        return float(torch.linalg.norm(u - v) / torch.linalg.norm(v))

    assert rel(f, fr) < tol
    for u, v in zip(got, ref):
        assert rel(u, v) < tol
