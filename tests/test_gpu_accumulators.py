"""P1 launches on cells in no order, in part or throughout, against the oracle: tiles that exceed
the accumulators, and the launch over every tile pair that operators of one space take where the
matrix exceeds L2."""

import numpy as np
import pytest

from bempp import shapes
from bempp.assembly.boundary import BoundaryAssemblerOptions, create_laplace_assembler
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndelement.reference_cell import ReferenceCellType
from ndgrid.grid import Grid

from test_gpu_parity import FP64_TOL, OPS, SPACES, gpu_assemble, oracle_assemble, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [6, 16])
@pytest.mark.parametrize("kernel,op,sp", [("laplace", "double_layer", "p1"),
                                          ("laplace", "hypersingular", "p1"),
                                          ("helmholtz", "adjoint_double_layer", "p1"),
                                          ("helmholtz", "hypersingular", "p1"),
                                          ("helmholtz", "single_layer", "dp1")])
def test_tiles_of_both_kinds_in_one_launch(kernel, op, sp, q):
    """A mesh in a good order but for its last two tiles, whose cells are far apart."""
    points, cells = shapes.icosphere(3)
    cells = np.array(cells)
    order = np.random.default_rng(2).permutation(len(cells))
    tail = np.sort(order[:64])
    cells = np.concatenate([np.delete(cells, tail, axis=0), cells[order[:64]]])
    grid = Grid(shapes.radial_perturbation(points, seed=9), cells)
    a = gpu_assemble(grid, kernel, op, 3.0, SPACES[sp], q=q, one_space=True)
    assert rel_err(a, oracle_assemble(grid, kernel, op, 3.0, SPACES[sp], SPACES[sp], q=q)) <= FP64_TOL


@pytest.mark.parametrize("op,host", [("hypersingular", False), ("hypersingular", True),
                                     ("adjoint_double_layer", False)])
def test_shuffled_cells_and_a_matrix_beyond_l2(op, host):
    """8,192 shuffled triangles, 134 MB: the device call in one launch and, where it covers half of
    the tile pairs too, the host call in chunks."""
    import torch

    points, cells = shapes.regular_sphere(5)
    cells = np.array(cells)[np.random.default_rng(3).permutation(len(cells))]
    grid = Grid(points, cells)
    space = function_space(grid, create_family(Family.Lagrange, 1, Continuity.Standard))
    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, 6)
    a = create_laplace_assembler(OPS[op], opts)
    if host:
        m = a.assemble(space, space)
    else:
        n = space.global_size
        out = torch.empty((n, n), dtype=torch.float64, device="cuda")
        a.assemble_into_device(space, space, out, torch.cuda.current_stream().cuda_stream)
        m = out.cpu().numpy().T
    assert rel_err(m, oracle_assemble(grid, "laplace", op, 0.0, SPACES["p1"], SPACES["p1"])) <= FP64_TOL
