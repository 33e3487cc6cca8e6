"""The singular part as directions and radii against the oracle's point by point sums: every
kernel and pairing of spaces, Duffy orders from 1 up, and wavenumbers that take each number
of series terms and the phases beyond the series.  The sums are the oracle's in another
order, so the FP64 tolerance of the parity tests applies."""

import numpy as np
import pytest

from bempp import shapes
from bempp.assembly.boundary import (BoundaryAssemblerOptions, create_helmholtz_assembler,
                                     create_laplace_assembler)
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndelement.reference_cell import ReferenceCellType
from ndgrid.grid import Grid

from test_gpu_parity import FP64_TOL, OPS, SPACES, oracle_assemble, rel_err

pytestmark = pytest.mark.gpu


def singular(grid, kernel, op, k, test, trial, order):
    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, 6)
    opts.set_singular_quadrature_degree(ReferenceCellType.Triangle, ReferenceCellType.Triangle, order)
    a = (create_laplace_assembler(OPS[op], opts) if kernel == "laplace"
         else create_helmholtz_assembler(OPS[op], k, opts))

    def space(sp):
        return function_space(grid, create_family(
            Family.Lagrange, SPACES[sp][0],
            Continuity.Standard if SPACES[sp][1] else Continuity.Discontinuous))

    return a.assemble_singular(space(trial), space(test)).toarray()


def check(kernel, op, k, test, trial, order, level=1):
    points, cells = shapes.icosphere(level)
    grid = Grid(shapes.radial_perturbation(points, seed=17), cells)
    a = singular(grid, kernel, op, k, test, trial, order)
    o = oracle_assemble(grid, kernel, op, k, SPACES[test], SPACES[trial], order=order, parts=2)
    assert rel_err(a, o) <= FP64_TOL


@pytest.mark.parametrize("order", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("kernel,k", [("laplace", 0.0), ("helmholtz", 0.6)])
@pytest.mark.parametrize("op,sp", [("single_layer", "p1"), ("double_layer", "p1"),
                                   ("hypersingular", "p1"), ("adjoint_double_layer", "dp0")])
def test_orders(order, kernel, k, op, sp):
    check(kernel, op, k, sp, sp, order)


# longest edge about 0.6 (80 cells): k times two diameters around 0.17, 0.5, 1.3, 3.3 and beyond
@pytest.mark.parametrize("k", [0.0, 0.1, 0.35, 1.0, 2.5, 3.2, 12.0])
@pytest.mark.parametrize("op", ["single_layer", "double_layer", "adjoint_double_layer"])
@pytest.mark.parametrize("test,trial", [("dp0", "dp0"), ("p1", "p1"), ("dp0", "p1"), ("p1", "dp0")])
def test_wavenumbers_and_spaces(k, op, test, trial):
    check("helmholtz", op, k, test, trial, 4)


@pytest.mark.parametrize("k", [0.1, 1.0, 2.5, 12.0])
def test_hypersingular_wavenumbers(k):
    check("helmholtz", "hypersingular", k, "p1", "p1", 4)


@pytest.mark.parametrize("op,sp", [("single_layer", "dp0"), ("double_layer", "p1")])
def test_one_thread_per_pair(op, sp):
    """Enough pairs (80,000 and more) that each has one thread."""
    check("helmholtz", op, 3.0, sp, sp, 2, level=4)
