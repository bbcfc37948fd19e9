"""Performance cases of the MD engine, through its public Python entry points.

A case is a dict of plain values; `prepare` builds the inputs and the engine
context that a program holds, `run` makes one pass, `work` counts what a pass
cannot do without and `exact` gives the same outputs from plain torch in 64
bits.  Four kinds of work:

  md         a box of atoms set on the device, Verlet setup, `steps` NVE steps
             with thermo rows, the final state read back on the device
  replicas   the same for a batch of independent uneven boxes
  snapshot   one configuration: neighbor list, forces, per-atom energy and
             virial (what a rerun or an analysis asks for each frame)
  match      force matching: forces of a trial force field, the loss against
             target forces, and its gradients (positions, epsilon, sigma)

Boxes are fcc lattices with Gaussian displacements, a fraction of the sites
left empty (odd atom counts), and Gaussian velocities.  Mixed-precision cases
fix the threads per atom, as a program that wants reproducible FP32 sums does;
FP64 cases leave the launch shape to the engine's search.
"""
import math

import numpy as np
import torch

DEV = "cuda:0"
CU_U3 = "tests/golden/Cu_u3.eam"
A_CU, MASS_CU = 3.615, 63.55
METAL = dict(boltz=8.617343e-5, mvv2e=1.0364269e-4, ftm2v=1.0 / 1.0364269e-4, nktv2p=1.6021765e6)
LJ = dict(boltz=1.0, mvv2e=1.0, ftm2v=1.0, nktv2p=1.0)
MAX_ATOM_STEPS = 4_000_000 * 60  # the largest listed case


def _md(name, style, precision, cells, steps, *, every=20, delay=0, check=False, lanes=0, thermo=0,
        holes=0.0, temp=1.44, types=1):
    nx, ny, nz = cells
    return dict(name=name, kind="md", style=style, precision=precision, nx=nx, ny=ny, nz=nz,
                steps=steps, every=every, delay=delay, check=check, lanes=lanes, thermo=thermo,
                holes=holes, temp=temp, types=types)


def listed():
    return [
        # a small melt, 864 atoms: every step is a few microseconds, launches decide
        _md("lj_864_mixed", "lj", "mixed", (6, 6, 6), 100, lanes=8, thermo=50),
        # the melt example's 4,000 atoms in the FP64 form, an output row every 50 steps
        _md("lj_4k_fp64", "lj", "fp64", (10, 10, 10), 200, thermo=50),
        # the 32,000-atom Lennard-Jones benchmark in both forms
        _md("lj_32k_mixed", "lj", "mixed", (20, 20, 20), 100, lanes=4, thermo=100),
        _md("lj_32k_fp64", "lj", "fp64", (20, 20, 20), 100, thermo=100),
        # the 32,000-atom copper benchmark (distance-checked lists, skin 1.0)
        _md("eam_32k_mixed", "eam", "mixed", (20, 20, 20), 100, every=1, delay=5, check=True,
            lanes=4, thermo=50, temp=1600.0),
        # a large metal box in FP64, uneven edges, vacancies (odd atom count)
        _md("eam_250k_fp64", "eam", "fp64", (36, 40, 44), 40, every=1, delay=5, check=True,
            holes=0.002, temp=1600.0),
        # a large FP64 fluid, uneven edges, two types, distance-checked lists
        _md("lj_500k_fp64", "lj", "fp64", (47, 50, 53), 40, every=10, check=True, holes=0.005,
            types=2),
        # the 4,000,000-atom Lennard-Jones headline box, mixed precision
        _md("lj_4m_mixed", "lj", "mixed", (100, 100, 100), 60, lanes=1),
        # a parameter sweep: 256 uneven boxes (500 to 6,912 atoms) advanced together
        dict(name="replicas_256_mixed", kind="replicas", precision="mixed", nrep=256, nlo=5, nhi=12,
             steps=60, lanes=1),
        # one frame of a three-type fluid in an uneven box with per-atom tallies
        dict(name="snapshot_109k_mixed", kind="snapshot", precision="mixed", nx=27, ny=30, nz=34,
             holes=0.01, types=3, lanes=4),
        # the two-type force-matching box: one forward and backward pass
        dict(name="match_8k_mixed", kind="match", precision="mixed", nx=10, ny=10, nz=20, holes=0.0,
             types=2),
        # a larger training frame in FP64, three types, odd atom count
        dict(name="match_55k_fp64", kind="match", precision="fp64", nx=23, ny=24, nz=25, holes=0.01,
             types=3),
    ]


def _cells(rng, lo, hi):
    """An uneven fcc block of about log-uniform lo..hi atoms."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    edge = (n / 4.0) ** (1.0 / 3.0)
    return [max(5, round(edge * rng.uniform(0.9, 1.1))) for _ in range(3)]


def _lanes(precision, n):
    """Threads per atom of a mixed case: about what the search picks at this size."""
    if precision != "mixed":
        return 0
    return 8 if n < 12_000 else 4 if n < 120_000 else 2 if n < 400_000 else 1


def draw(rng):
    kind = rng.choice(["md", "md", "md", "md", "replicas", "snapshot", "match", "match"])
    precision = rng.choice(["mixed", "fp64"])
    if kind == "md":
        style = rng.choice(["lj", "lj", "eam"])
        nx, ny, nz = _cells(rng, 500, 1_500_000 if style == "lj" else 300_000)
        if style == "lj" and rng.random() < 0.6:
            ny = nz = nx  # most fluids sit in cubes
        n = 4 * nx * ny * nz
        steps = min(rng.randint(20, 150), max(20, MAX_ATOM_STEPS // (2 * n)))
        check = style == "eam" or rng.random() < 0.3
        c = _md("", style, precision, (nx, ny, nz), steps,
                every=rng.choice([1, 5]) if check else rng.choice([10, 20]),
                delay=5 if check else 0, check=check, lanes=_lanes(precision, n),
                thermo=rng.choice([0, 10, 50]), holes=rng.choice([0.0, 0.003, 0.02]),
                temp=round(rng.uniform(300.0, 1600.0), 1) if style == "eam"
                else round(rng.uniform(0.8, 2.0), 3),
                types=1 if style == "eam" else rng.choice([1, 1, 2, 3]))
        del c["name"]
        return c
    if kind == "replicas":
        return dict(kind=kind, precision=precision, nrep=rng.randint(12, 256), nlo=5,
                    nhi=rng.randint(7, 12), steps=rng.randint(20, 60),
                    lanes=1 if precision == "mixed" else 0)
    nx, ny, nz = _cells(rng, 1_000, 150_000 if kind == "snapshot" else 80_000)
    c = dict(kind=kind, precision=precision, nx=nx, ny=ny, nz=nz,
             holes=rng.choice([0.0, 0.01, 0.03]), types=rng.randint(1, 4))
    if kind == "snapshot":
        c["lanes"] = _lanes(precision, 4 * nx * ny * nz)
    return c


# ---- inputs -----------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1_000_003 * (seed + 1) % (2**31))
    return g


def _fcc(nx, ny, nz, a, jitter, holes, g):
    """Positions (n, 3) in creation order and the box edges."""
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]],
                         dtype=torch.float64, device=DEV)
    k, j, i = torch.meshgrid(*(torch.arange(m, device=DEV, dtype=torch.float64)
                               for m in (nz, ny, nx)), indexing="ij")
    x = (torch.stack([i, j, k], -1).reshape(-1, 1, 3) + basis).reshape(-1, 3) * a
    x = x + jitter * torch.randn(x.shape, generator=g, device=DEV, dtype=torch.float64)
    edge = torch.tensor([nx * a, ny * a, nz * a], dtype=torch.float64, device=DEV)
    x = torch.remainder(x, edge)
    x = torch.where(x >= edge, torch.zeros_like(x), x)
    if holes > 0:
        n = x.shape[0]
        keep = n - max(1, int(holes * n))
        keep -= 1 - keep % 2  # an odd count
        x = x[torch.randperm(n, generator=g, device=DEV)[:keep].sort().values]
    return x.contiguous(), edge


def _velocities(n, temp, mass, u, g):
    v = torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float64)
    v = v - v.mean(0)
    t = u["mvv2e"] * mass * (v * v).sum() / ((3 * n - 3) * u["boltz"])
    return (v * torch.sqrt(temp / t)).contiguous()


def _types(n, ntypes, g):
    return (torch.randint(0, ntypes, (n,), generator=g, device=DEV) + 1).to(torch.int32)


def _lattice_constant(rho):
    return (4.0 / rho) ** (1.0 / 3.0)


def _lj_coeffs(ntypes):
    """Diagonal epsilon and sigma; the cross terms mix geometrically, rc = 2.5 sigma."""
    return [(1.0, 1.0), (0.8, 0.95), (1.2, 1.04), (0.9, 0.98)][:ntypes]


def _system(case, n_types, lo, hi):
    from lammps_b200 import PairEAM, PairLJCut, System

    eam = case.get("style") == "eam"
    s = System("metal" if eam else "lj", case["precision"])
    s.set_box(lo, hi)
    if eam:
        p = PairEAM(1)
        p.coeff(1, CU_U3)
        s.set_pair(p)
    else:
        p = PairLJCut(2.5, n_types)
        for t, (e, sg) in enumerate(_lj_coeffs(n_types), start=1):
            p.coeff(t, t, e, sg, 2.5 * sg)
        s.set_pair(p)
        s.set_mass([1.0 + 0.25 * t for t in range(n_types)])
    s.set_neighbor(1.0 if eam else 0.3, case.get("every", 20), case.get("delay", 0),
                   case.get("check", False))
    s.set_timestep(0.005)
    s.set_thermo(case.get("thermo", 0))
    if case.get("lanes"):
        s.set_launch(case["lanes"])
    return s


def _replica_edges(case):
    """Unit cells per edge of each replica: log-uniform atom counts, the same for every seed."""
    rng = np.random.default_rng(20140808 + 100 * case["nrep"] + case["nhi"])
    target = np.exp(rng.uniform(np.log(500), np.log(4 * case["nhi"] ** 3), case["nrep"]))
    return np.clip(np.round((target / 4.0) ** (1 / 3)), case["nlo"], case["nhi"]).astype(int)


def _inputs(case, seed):
    """The arrays of a case on the GPU, from the seed alone."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "replicas":
        rng = np.random.default_rng(seed + 77)
        edge, nrep = _replica_edges(case), case["nrep"]
        rho, temp = rng.uniform(0.70, 0.95, nrep), rng.uniform(0.8, 2.0, nrep)
        xs, vs, hi = [], [], []
        for r in range(nrep):
            e = int(edge[r])
            x, L = _fcc(e, e, e, _lattice_constant(rho[r]), 0.03, 0.0, g)
            xs.append(x)
            vs.append(_velocities(len(x), float(temp[r]), 1.0, LJ, g))
            hi.append(L.cpu().numpy())
        x = torch.cat(xs)
        return dict(x=x, v=torch.cat(vs), type=torch.ones(len(x), dtype=torch.int32, device=DEV),
                    natoms=np.array([len(q) for q in xs], np.int32), hi=np.array(hi))
    eam = case.get("style") == "eam"
    a = A_CU if eam else _lattice_constant(0.85 if kind == "match" else 0.8442)
    x, edge = _fcc(case["nx"], case["ny"], case["nz"], a, 0.05, case["holes"], g)
    d = dict(x=x, edge=edge, type=_types(len(x), case.get("types", 1), g))
    if kind == "md":
        d["v"] = _velocities(len(x), case["temp"], MASS_CU if eam else 1.0, METAL if eam else LJ, g)
    if kind == "match":
        r = np.random.default_rng(seed + 4242)
        m = case["types"] * (case["types"] + 1) // 2
        d["eps"], d["sigma"] = r.uniform(0.5, 1.5, m), r.uniform(0.9, 1.1, m)
        # the trial parameters, off the hidden ones that made the targets
        d["eps0"] = d["eps"] * (1 + 0.08 * r.standard_normal(m))
        d["sigma0"] = d["sigma"] * (1 + 0.02 * r.standard_normal(m).clip(-2, 2))
    return d


MATCH_CUT = 2.5 * 1.1 * 1.05


def _match_target(case, d):
    """Forces at the hidden parameters, in plain torch."""
    t = d["type"].long()
    i, j = _pairs(d["x"], [(0, len(t), d["edge"])], MATCH_CUT)
    e, s = (_matrix(torch.as_tensor(d[k], device=DEV), case["types"]) for k in ("eps", "sigma"))
    return _lj_forces(d["x"], d["edge"], i, j, t, 48 * e * s**12, 24 * e * s**6, (2.5 * s) ** 2)


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "match":
        from lammps_b200.forcematch import LJForceField

        lo = np.zeros(3)
        ff = LJForceField(lo, d["edge"].cpu().numpy(), d["x"].cpu().numpy(),
                          d["type"].cpu().numpy(), case["types"], MATCH_CUT, case["precision"])
        leaf = lambda k: torch.tensor(d[k], dtype=torch.float64, requires_grad=True)  # noqa: E731
        return dict(kind=kind, ff=ff, x=d["x"].clone().requires_grad_(True), eps=leaf("eps0"),
                    sigma=leaf("sigma0"), target=_match_target(case, d), ntypes=case["types"])
    if kind == "replicas":
        from lammps_b200.replicas import make_batch

        s = make_batch(dict(x=d["x"].cpu().numpy(), v=d["v"].cpu().numpy(), natoms=d["natoms"],
                            lo=np.zeros_like(d["hi"]), hi=d["hi"]), case["precision"],
                       tpa=case["lanes"])
        s.set_replica_step(1)  # a graph of kernels per step: one FP32 summation order
        s.setup()
        return dict(kind=kind, s=s, x=d["x"], v=d["v"], type=d["type"], steps=case["steps"])
    s = _system(case, case.get("types", 1), np.zeros(3), d["edge"].cpu().numpy())
    st = dict(kind=kind, s=s, x=d["x"], v=d.get("v"), type=d["type"], steps=case.get("steps"))
    s.set_atoms_dev(st["x"], st["type"], st["v"])
    if kind == "md":
        s.setup()  # the context's buffers and launch shape
    else:
        s.neigh_build()
    return st


# ---- one pass ---------------------------------------------------------------


def _rows(rows):
    return np.array([[r["Temp"], r["E_pair"], r["TotEng"], r["Press"]] for r in rows])


def run(state):
    kind = state["kind"]
    if kind == "match":
        from lammps_b200.forcematch import pair_matrix

        nt = state["ntypes"]
        f = state["ff"].forces(state["x"], pair_matrix(state["eps"], nt),
                               pair_matrix(state["sigma"], nt))
        loss = ((f - state["target"]) ** 2).sum(dim=1).mean()
        gx, ge, gs = torch.autograd.grad(loss, (state["x"], state["eps"], state["sigma"]))
        return dict(f=f.detach(), loss=loss.detach(), gx=gx, geps=ge, gsigma=gs)
    s = state["s"]
    s.set_atoms_dev(state["x"], state["type"], state["v"])
    if kind == "snapshot":
        s.neigh_build()
        tally = s.compute_dev()
        out = s.download_dev(f=True)
        return dict(f=out["f"], eatom=tally["eatom"], vatom=tally["vatom"])
    first = s.setup()
    rows = s.run(state["steps"])
    out = s.download_dev(f=True)
    if kind == "md":
        out["thermo"] = _rows([first] + rows)
    else:
        out["thermo"] = _rows(s.replica_thermo())
    return out


# ---- what a pass cannot do without ------------------------------------------


def _atoms(case):
    if case["kind"] == "replicas":
        return int((4 * _replica_edges(case) ** 3).sum())
    n = 4 * case["nx"] * case["ny"] * case["nz"]
    if case["holes"] > 0:
        n -= max(1, int(case["holes"] * n))
        n -= 1 - n % 2
    return n


def work(case):
    """Inputs read once and outputs written once; pair arithmetic of the half
    pairs inside the cutoff (27 at 2.5 sigma, 21 in copper), no list, no skin."""
    n, kind = _atoms(case), case["kind"]
    if kind == "match":
        # x, types, targets in; forces and dL/dx out; a forward and an adjoint term per pair
        return dict(bytes=n * (24 + 4 + 24 + 24 + 24), flops=n * 27 * (27 + 75))
    if kind == "snapshot":
        return dict(bytes=n * (24 + 4 + 24 + 8 + 48), flops=n * (27 * 45 + 15))
    per_step = 1695 if case.get("style") == "eam" else 745
    return dict(bytes=n * (48 + 4 + 72 + 12), flops=n * per_step * (case["steps"] + 1))


# ---- the same outputs in plain torch, 64 bits ---------------------------------


def _matrix(values, ntypes):
    m = torch.zeros((ntypes + 1, ntypes + 1), dtype=values.dtype, device=values.device)
    r = [i for i in range(1, ntypes + 1) for j in range(i, ntypes + 1)]
    c = [j for i in range(1, ntypes + 1) for j in range(i, ntypes + 1)]
    r, c = (torch.tensor(q, device=values.device) for q in (r, c))
    return m.index_put((r, c), values).index_put((c, r), values)


def _box_pairs(x, edge, cut):
    """Directed pairs (i, j) within cut at the minimum image of one box."""
    n = len(x)
    nc = torch.clamp((edge / cut).long(), min=1)
    ii, jj = [], []
    if int(nc.min()) < 3 or n < 2000:
        for a in range(0, n, 4096):
            d = x[a:a + 4096, None] - x[None]
            d = d - edge * torch.round(d / edge)
            p = ((d * d).sum(-1) <= cut * cut).nonzero()
            ii.append(p[:, 0] + a)
            jj.append(p[:, 1])
    else:
        w = torch.remainder(x, edge)
        c = torch.minimum((w / edge * nc).long(), nc - 1)
        cid = c[:, 0] + nc[0] * (c[:, 1] + nc[1] * c[:, 2])
        m = int(nc.prod())
        cnt = torch.bincount(cid, minlength=m)
        start = torch.cumsum(cnt, 0) - cnt
        order = torch.argsort(cid)
        width = int(cnt.max())
        slot = torch.empty_like(cid)
        slot[order] = torch.arange(n, device=x.device) - start[cid[order]]
        table = torch.full((m, width), -1, dtype=torch.long, device=x.device)
        table[cid, slot] = torch.arange(n, device=x.device)
        block = max(1, 40_000_000 // (27 * width))
        off = torch.cartesian_prod(*(torch.tensor([-1, 0, 1], device=x.device),) * 3)
        for a in range(0, n, block):
            q = torch.remainder(c[a:a + block, None] + off, nc)
            j = table[q[..., 0] + nc[0] * (q[..., 1] + nc[1] * q[..., 2])].reshape(len(q), -1)
            d = x[a:a + block, None] - x[j.clamp(min=0)]
            d = d - edge * torch.round(d / edge)
            p = ((j >= 0) & ((d * d).sum(-1) <= cut * cut)).nonzero()
            ii.append(p[:, 0] + a)
            jj.append(j[p[:, 0], p[:, 1]])
    i, j = torch.cat(ii), torch.cat(jj)
    keep = i != j
    return i[keep], j[keep]


def _pairs(x, boxes, cut):
    got = [_box_pairs(x[a:b], edge, cut) for a, b, edge in boxes]
    return (torch.cat([i + b[0] for (i, _), b in zip(got, boxes)]),
            torch.cat([j + b[0] for (_, j), b in zip(got, boxes)]))


def _separations(x, edge, i, j):
    d = x[i] - x[j]
    L = edge if edge.dim() == 1 else edge[i]
    return d - L * torch.round((d / L).detach())


def _lj_forces(x, edge, i, j, t, lj1, lj2, cutsq):
    d = _separations(x, edge, i, j)
    r2 = (d * d).sum(-1)
    tt = (t[i], t[j])
    r6 = 1.0 / r2**3
    w = torch.where(r2 < cutsq[tt], (lj1[tt] * r6 - lj2[tt]) * r6 / r2, torch.zeros_like(r2))
    return torch.zeros_like(x).index_add(0, i, d * w[:, None])


def _lj_tables(ntypes):
    e, s = (torch.zeros((ntypes + 1, ntypes + 1), dtype=torch.float64, device=DEV) for _ in "es")
    co = _lj_coeffs(ntypes)
    for a in range(ntypes):
        for b in range(ntypes):
            e[a + 1, b + 1] = math.sqrt(co[a][0] * co[b][0])
            s[a + 1, b + 1] = math.sqrt(co[a][1] * co[b][1])
    return e, s


class _LJField:
    def __init__(self, ntypes, t):
        self.e, self.s = _lj_tables(ntypes)
        self.t, self.cut = t, 2.5 * float(self.s.max())

    def __call__(self, x, edge, i, j):
        """Forces, per-atom energy and per-atom virial (n, 6)."""
        d = _separations(x, edge, i, j)
        r2 = (d * d).sum(-1)
        tt = (self.t[i], self.t[j])
        e, s = self.e[tt], self.s[tt]
        near = r2 < (2.5 * s) ** 2
        d, r2, e, s, i = d[near], r2[near], e[near], s[near], i[near]
        q = (s * s / r2) ** 3
        w = 24 * e * q * (2 * q - 1) / r2
        f = torch.zeros_like(x).index_add(0, i, d * w[:, None])
        ea = torch.zeros_like(x[:, 0]).index_add(0, i, 2 * e * q * (q - 1))
        return f, ea, _virial(x, d, w, i)


def _virial(x, d, w, i):
    h = 0.5 * w
    cols = [d[:, a] * d[:, b] * h for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
    return torch.zeros((len(x), 6), dtype=x.dtype, device=x.device).index_add(
        0, i, torch.stack(cols, 1))


def _spline(delta, f):
    """The 7-coefficient cubic of the embedded-atom tables at knots 0..n-1."""
    n = len(f)
    c = np.zeros((n, 7))
    c[:, 6] = f
    c[0, 5], c[1, 5] = f[1] - f[0], 0.5 * (f[2] - f[0])
    c[n - 2, 5], c[n - 1, 5] = 0.5 * (f[n - 1] - f[n - 3]), f[n - 1] - f[n - 2]
    c[2:n - 2, 5] = ((f[:n - 4] - f[4:]) + 8.0 * (f[3:n - 1] - f[1:n - 3])) / 12.0
    df = f[1:] - f[:-1]
    c[:-1, 4] = 3.0 * df - 2.0 * c[:-1, 5] - c[1:, 5]
    c[:-1, 3] = c[:-1, 5] + c[1:, 5] - 2.0 * df
    c[:, 2], c[:, 1], c[:, 0] = c[:, 5] / delta, 2.0 * c[:, 4] / delta, 3.0 * c[:, 3] / delta
    return torch.tensor(c, device=DEV)


def _eval(c, p, lowest=0):
    """Value and derivative of a spline at fractional knot p (0-based)."""
    m = p.long().clamp(lowest, len(c) - 2)
    p = (p - m).clamp(max=1.0)
    k = c[m]
    return (((k[:, 3] * p + k[:, 4]) * p + k[:, 5]) * p + k[:, 6],
            (k[:, 0] * p + k[:, 1]) * p + k[:, 2])


class _EAMField:
    def __init__(self):
        with open(CU_U3) as fh:
            lines = fh.read().splitlines()
        h = lines[2].split()
        nrho, self.drho, nr, self.dr = int(h[0]), float(h[1]), int(h[2]), float(h[3])
        self.cut = float(h[4])
        v = np.array([float(t) for line in lines[3:] for t in line.split()])
        # the common grid of one file has one knot less than the file
        nf, ng = int((nrho - 1) * self.drho / self.drho + 0.5), int((nr - 1) * self.dr / self.dr + 0.5)
        self.F = _spline(self.drho, v[:nf])
        self.z2 = _spline(self.dr, 27.2 * 0.529 * v[nrho:nrho + ng] ** 2)
        self.rho = _spline(self.dr, v[nrho + nr:nrho + nr + ng])
        self.rhomax = (nrho - 1) * self.drho

    def __call__(self, x, edge, i, j):
        d = _separations(x, edge, i, j)
        r2 = (d * d).sum(-1)
        near = r2 < self.cut**2
        d, r, i, j = d[near], r2[near].sqrt(), i[near], j[near]
        p = r / self.dr
        rho, drho = _eval(self.rho, p)
        total = torch.zeros_like(x[:, 0]).index_add(0, i, rho)
        F, dF = _eval(self.F, total / self.drho)
        F = F + torch.where(total > self.rhomax, dF * (total - self.rhomax), torch.zeros_like(F))
        z2, dz2 = _eval(self.z2, p)
        phi = z2 / r
        psi = (dF[i] + dF[j]) * drho + (dz2 - phi) / r
        w = -psi / r
        f = torch.zeros_like(x).index_add(0, i, d * w[:, None])
        return f, F.index_add(0, i, 0.5 * phi), _virial(x, d, w, i)


def _thermo_row(n, vol, ke2, pe, vir, u, per_atom):
    dof = 3.0 * n - 3.0
    temp = u["mvv2e"] * ke2 / (dof * u["boltz"])
    ke = 0.5 * dof * u["boltz"] * temp
    press = (dof * u["boltz"] * temp + vir) / 3.0 / vol * u["nktv2p"]
    k = n if per_atom else 1
    return [temp, pe / k, (pe + ke) / k, press]


def _exact_run(case, d):
    eam = case.get("style") == "eam"
    u, dt = (METAL if eam else LJ), 0.005
    replicas = case["kind"] == "replicas"
    t = d["type"].long()
    n = len(t)
    if replicas:
        ends = np.cumsum(d["natoms"])
        boxes = [(int(b - k), int(b), torch.tensor(hi, device=DEV))
                 for b, k, hi in zip(ends, d["natoms"], d["hi"])]
        edge = torch.cat([e.expand(b - a, 3) for a, b, e in boxes])
    else:
        boxes, edge = [(0, n, d["edge"])], d["edge"]
    nt = case.get("types", 1)
    field = _EAMField() if eam else _LJField(nt, t)
    m = torch.full((n, 1), MASS_CU, dtype=torch.float64, device=DEV) if eam else \
        (1.0 + 0.25 * (t - 1).double())[:, None]
    skin = 1.0 if eam else 0.3
    every, delay, check = case.get("every", 20), case.get("delay", 0), case.get("check", False)
    x, v = d["x"].clone(), d["v"].clone()
    image = torch.zeros((n, 3), dtype=torch.int32, device=DEV)
    dtfm = 0.5 * dt * u["ftm2v"] / m

    def build():
        nonlocal x, image
        up, down = x >= edge, x < 0
        x = x + edge * down - edge * up
        image = image + up.int() - down.int()
        if nt == 1:
            i, j = _pairs(x, boxes, field.cut + skin)
        else:  # per-type list cutoffs
            i, j = _pairs(x, boxes, field.cut + skin)
            s = _separations(x, edge, i, j)
            near = (s * s).sum(-1) <= (2.5 * field.s[t[i], t[j]] + skin) ** 2
            i, j = i[near], j[near]
        return i, j, x

    def rows(f, ea, va):
        out = []
        for a, b, e in boxes:
            k2 = float((m[a:b] * v[a:b] ** 2).sum())
            out.append(_thermo_row(b - a, float(e.prod()), k2, float(ea[a:b].sum()),
                                   float(va[a:b, :3].sum()), u, not eam))
        return out

    i, j, hold = build()
    f, ea, va = field(x, edge, i, j)
    thermo, ago = rows(f, ea, va), 0
    for step in range(1, case["steps"] + 1):
        v = v + dtfm * f
        x = x + dt * v
        ago += 1
        if ago >= delay and ago % every == 0 and (
                not check or float(((x - hold) ** 2).sum(-1).max()) > 0.25 * skin * skin):
            i, j, hold = build()
            ago = 0
        f, ea, va = field(x, edge, i, j)
        v = v + dtfm * f
        last = step == case["steps"]
        if replicas:
            if last:
                thermo = rows(f, ea, va)
        elif last or (case["thermo"] and step % case["thermo"] == 0):
            thermo += rows(f, ea, va)
    return dict(x=x, v=v, image=image, f=f, thermo=np.array(thermo))


def exact(case, seed):
    """`run`'s outputs in plain torch and 64 bits (the list schedule is the
    engine's: a pair that enters the cutoff between two builds is not seen);
    None for the boxes that take too long."""
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("md", "replicas"):
        if _atoms(case) * case["steps"] > 25_000_000:
            return None
        return _exact_run(case, d)
    t = d["type"].long()
    if kind == "snapshot":
        field = _LJField(case["types"], t)
        i, j = _pairs(d["x"], [(0, len(t), d["edge"])], field.cut)
        f, ea, va = field(d["x"], d["edge"], i, j)
        return dict(f=f, eatom=ea, vatom=va)
    target = _match_target(case, d)
    x = d["x"].clone().requires_grad_(True)
    eps, sigma = (torch.tensor(d[k], dtype=torch.float64, device=DEV, requires_grad=True)
                  for k in ("eps0", "sigma0"))
    e, s = _matrix(eps, case["types"]), _matrix(sigma, case["types"])
    with torch.no_grad():
        i, j = _pairs(d["x"], [(0, len(t), d["edge"])], MATCH_CUT)
    f = _lj_forces(x, d["edge"], i, j, t, 48 * e * s**12, 24 * e * s**6, (2.5 * s.detach()) ** 2)
    loss = ((f - target) ** 2).sum(dim=1).mean()
    gx, ge, gs = torch.autograd.grad(loss, (x, eps, sigma))
    return dict(f=f.detach(), loss=loss.detach(), gx=gx, geps=ge, gsigma=gs)
