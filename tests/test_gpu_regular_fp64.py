"""The FP64 regular kernels at the edges of their dispatch, against the oracle: cell counts
around the 32-cell tile, the 16-cell chunk and the four test tiles of a block; the 6-point
rule and the general form (remainders of its groups of test points, the test points split
over the warps); accumulators that fit in shared memory and those that do not (shuffled
cells: up to 96 DOFs per tile); both phase forms.  Same rules and formulas as the oracle, so
the FP64 tolerance of the parity tests applies."""

import numpy as np
import pytest

from bempp import shapes
from ndgrid.grid import Grid

from test_gpu_parity import FP64_TOL, SPACES, gpu_assemble, oracle_assemble, rel_err

pytestmark = pytest.mark.gpu


def surface(ncells, shuffled=False):
    """The first ncells cells of a perturbed icosphere (closed when that is all of them)."""
    level = 0
    while 20 * 4 ** level < ncells:
        level += 1
    points, cells = shapes.icosphere(level)
    points = shapes.radial_perturbation(points, seed=5)
    cells = cells[:ncells]
    if shuffled:
        cells = cells[np.random.default_rng(3).permutation(ncells)]
    used = np.unique(cells)
    remap = np.zeros(len(points), dtype=np.int64)
    remap[used] = np.arange(len(used))
    return Grid(points[used], remap[cells])


@pytest.mark.parametrize("ncells", [31, 33, 129, 161])
@pytest.mark.parametrize("kernel,op,k,sp", [("laplace", "double_layer", 0.0, "p1"),
                                            ("laplace", "hypersingular", 0.0, "p1"),
                                            ("helmholtz", "single_layer", 9.0, "dp0"),
                                            ("helmholtz", "adjoint_double_layer", 0.7, "p1")])
def test_sizes_around_the_tiles(ncells, kernel, op, k, sp):
    grid = surface(ncells)
    a = gpu_assemble(grid, kernel, op, k, SPACES[sp], one_space=True)
    assert rel_err(a, oracle_assemble(grid, kernel, op, k, SPACES[sp], SPACES[sp])) <= FP64_TOL


@pytest.mark.parametrize("q", [1, 3, 7, 19, 37])
@pytest.mark.parametrize("kernel,op,k,sp", [("laplace", "single_layer", 0.0, "dp0"),
                                            ("laplace", "adjoint_double_layer", 0.0, "p1"),
                                            ("helmholtz", "double_layer", 6.0, "p1"),
                                            ("helmholtz", "hypersingular", 1.0, "p1")])
def test_general_rules(q, kernel, op, k, sp):
    grid = surface(97)
    a = gpu_assemble(grid, kernel, op, k, SPACES[sp], q=q, one_space=True)
    assert rel_err(a, oracle_assemble(grid, kernel, op, k, SPACES[sp], SPACES[sp], q=q)) <= FP64_TOL


@pytest.mark.parametrize("q", [6, 16])
@pytest.mark.parametrize("op", ["single_layer", "double_layer", "adjoint_double_layer",
                                "hypersingular"])
@pytest.mark.parametrize("sp", ["p1", "dp1"])
def test_blocks_without_shared_accumulators(op, sp, q):
    grid = surface(320, shuffled=True)
    a = gpu_assemble(grid, "helmholtz", op, 3.0, SPACES[sp], q=q, one_space=True)
    assert rel_err(a, oracle_assemble(grid, "helmholtz", op, 3.0, SPACES[sp], SPACES[sp], q=q)) <= FP64_TOL


def test_phases_beyond_any_reduction_stay_on_the_unit_circle():
    """k r of 1e17: its last digit is worth more than 2 pi, so the phase is arbitrary, but
    every kernel value must keep its modulus 1 / (4 pi r)."""
    grid = surface(80)
    far = np.linalg.norm(gpu_assemble(grid, "helmholtz", "single_layer", 1e17, one_space=True))
    still = np.linalg.norm(gpu_assemble(grid, "laplace", "single_layer", one_space=True))
    assert np.isfinite(far) and far <= still * (1.0 + 1e-9)
