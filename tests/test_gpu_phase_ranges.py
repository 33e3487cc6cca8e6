"""FP64 Helmholtz assembly with the 6-point rule on both sides of each limit of its phase forms:
the largest |k (r - r0)| of the mesh, bounded by 0.7253 circumradii on each side, just below and
just above 0.42 and 0.8.  Same rule and formulas as the oracle: the parity tests' tolerance."""

import numpy as np
import pytest

from test_gpu_parity import FP64_TOL, SPACES, gpu_assemble, oracle_assemble, rel_err
from test_gpu_regular_fp64 import surface

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0.42, 0.8])
@pytest.mark.parametrize("side", [0.999, 1.001])
@pytest.mark.parametrize("op,sp", [("single_layer", "dp0"), ("double_layer", "p1"),
                                   ("hypersingular", "p1")])
def test_around_the_limits(limit, side, op, sp):
    grid = surface(150)
    v = np.asarray(grid.points)[np.asarray(grid.cells)]
    rad = np.sqrt(((v - v.mean(axis=1, keepdims=True)) ** 2).sum(-1)).max()
    k = side * limit / (2 * 0.725270869 * rad)
    a = gpu_assemble(grid, "helmholtz", op, k, SPACES[sp], one_space=True)
    assert rel_err(a, oracle_assemble(grid, "helmholtz", op, k, SPACES[sp], SPACES[sp])) <= FP64_TOL
