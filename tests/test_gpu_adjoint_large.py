"""Force matching where one thread takes an atom: the smallest box of that
shape and the largest below it, by the comparison of the other shapes."""
import pytest

import test_gpu_adjoint_shapes as shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 1e-5)])
@pytest.mark.parametrize("cells,drop", [((25, 25, 18), 0), ((25, 25, 18), 1)])  # 45,000 atoms
def test_forward_backward(cells, drop, precision, tol):
    shapes.test_forward_backward(cells, 2, drop, precision, tol)
