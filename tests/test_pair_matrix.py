"""pair_matrix against its definition, element by element, with its derivatives
and under torch's transforms; and what it refuses."""
import pytest

torch = pytest.importorskip("torch")

from lammps_b200.forcematch import pair_matrix  # noqa: E402


def plain(values, ntypes):
    values = values.reshape(-1)
    at = {}
    for i in range(1, ntypes + 1):
        for j in range(i, ntypes + 1):
            at[i, j] = at[j, i] = len(set(at.values())) if (i, j) not in at else at[i, j]
    rows = [torch.stack([values[at[i, j]] if (i, j) in at else values.new_zeros(())
                         for j in range(ntypes + 1)]) for i in range(ntypes + 1)]
    return torch.stack(rows)


@pytest.mark.parametrize("ntypes", [1, 2, 3, 4, 7])
def test_values_and_derivatives(ntypes):
    k = ntypes * (ntypes + 1) // 2
    gen = torch.Generator().manual_seed(ntypes)
    v = torch.rand(k, dtype=torch.float64, generator=gen)
    g = torch.rand((ntypes + 1, ntypes + 1), dtype=torch.float64, generator=gen)
    assert torch.equal(pair_matrix(v, ntypes), plain(v, ntypes))
    for d in (torch.func.grad, torch.func.jacfwd, torch.func.hessian):
        got, want = (d(lambda q, m=m: (m(q, ntypes) ** 3 * g).sum())(v)
                     for m in (pair_matrix, plain))
        torch.testing.assert_close(got, want, rtol=1e-14, atol=0)
    b = torch.rand((5, k), dtype=torch.float64, generator=gen)
    many = torch.func.vmap(lambda q: pair_matrix(q, ntypes))(b)
    assert torch.equal(many, torch.stack([plain(q, ntypes) for q in b]))


def test_other_forms():
    assert torch.equal(pair_matrix(torch.tensor(5.0), 1), torch.tensor([[0.0, 0.0], [0.0, 5.0]]))
    every_other = torch.arange(6.0)[::2]  # not contiguous
    assert torch.equal(pair_matrix(every_other, 2), plain(every_other, 2))
    half = torch.tensor([1.0, 2.0, 3.0]).half()
    assert pair_matrix(half, 2).dtype == torch.float16


@pytest.mark.parametrize("shape,ntypes", [((3, 1), 2), ((1, 3), 2), ((1, 1), 1), ((2, 5), 4),
                                          ((0,), 0), ((0,), -1), ((2,), 2), ((4,), 2)])
def test_refused(shape, ntypes):
    with pytest.raises(ValueError):
        pair_matrix(torch.zeros(shape), ntypes)
