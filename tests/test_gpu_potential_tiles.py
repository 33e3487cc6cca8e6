"""The potential kernel at the edges of its tiles against the oracle: point counts around
the 32 points of a warp and the 128 of a block, cell counts around the 32-cell tile, rules
with remainders of the four-point groups, columns in shared memory (P1) and direct adds
(shuffled cells, degree 2).  Same rule and formulas, so the FP64 tolerance applies."""

import numpy as np
import pytest

from bempp import shapes
from bempp.assembly.boundary import BoundaryAssemblerOptions, OperatorType
from bempp.assembly.potential import (create_helmholtz_potential_assembler,
                                      create_laplace_potential_assembler)
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndelement.reference_cell import ReferenceCellType
from oracle import potential

from test_gpu_parity import FP64_TOL, rel_err
from test_gpu_regular_fp64 import surface

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npoints", [1, 31, 33, 129])
@pytest.mark.parametrize("ncells,q,shuffled", [(33, 6, False), (97, 7, False), (320, 3, True)])
@pytest.mark.parametrize("kernel,op,k,degree", [("laplace", "double_layer", 0.0, 0),
                                                ("laplace", "single_layer", 0.0, 1),
                                                ("helmholtz", "double_layer", 7.0, 1),
                                                ("helmholtz", "single_layer", 30.0, 2)])
def test_potential_tiles(npoints, ncells, q, shuffled, kernel, op, k, degree):
    grid = surface(ncells, shuffled)
    x = np.random.default_rng(npoints).standard_normal((npoints, 3))
    x *= 2.5 / np.linalg.norm(x, axis=1)[:, None]
    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, q)
    operator = OperatorType.DoubleLayer if op == "double_layer" else OperatorType.SingleLayer
    a = (create_laplace_potential_assembler(operator, opts) if kernel == "laplace"
         else create_helmholtz_potential_assembler(operator, k, opts))
    space = function_space(grid, create_family(
        Family.Lagrange, degree, Continuity.Standard if degree else Continuity.Discontinuous))
    p = a.assemble(space, x)
    o = potential.potential(x, grid.points, grid.cells.astype(np.int64), kernel, op, k=k,
                            degree=degree, continuous=degree > 0, q_regular=q)
    assert rel_err(p, o) <= FP64_TOL
