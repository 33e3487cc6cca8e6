"""Adjoint gradient at the edges of its 32-cell tiles and of its two phase forms.

Every coordinate derivative and dJ/dk against central differences (h = 1e-6) of
Re(lambda^H A mu) with A from the dense FP64 assembly.  Sizes: one partial tile (20 cells), tiles
and a remainder on a closed and on an open surface; k = 1 keeps every phase k (r - r0) of these
meshes' smaller tiles below 0.8, k = 25 none.  Tolerance, relative to the largest derivative:
the differences' rounding is about eps |J| / h <= 1e-9 of it and their truncation h^2 k^2 / 6 <= 1e-10,
so 1e-6 leaves the margin that the atomic sums and the entries' own errors need.
"""

import numpy as np
import pytest

from bempp import shapes
from bempp.assembly.boundary import (BoundaryAssemblerOptions, OperatorType,
                                     create_helmholtz_assembler)
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndelement.reference_cell import ReferenceCellType
from ndgrid.grid import Grid

pytestmark = pytest.mark.gpu


def surface(ncells):
    level = 0
    while 20 * 4 ** level < ncells:
        level += 1
    pts, cells = shapes.icosphere(level)
    pts, cells = shapes.radial_perturbation(pts, seed=ncells), np.asarray(cells)[:ncells]
    used, cells = np.unique(cells, return_inverse=True)
    return np.ascontiguousarray(pts[used]), cells.reshape(-1, 3)


def forward(pts, cells, k, lam, mu):
    import torch

    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, 6)
    a = create_helmholtz_assembler(OperatorType.SingleLayer, k, opts)
    sp = function_space(Grid(pts, cells), create_family(Family.Lagrange, 0, Continuity.Discontinuous))
    n = sp.global_size
    out = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    a.assemble_into_device(sp, sp, out, torch.cuda.current_stream().cuda_stream)
    return float(np.real(np.vdot(lam, out.cpu().numpy().T @ mu)))


@pytest.mark.parametrize("ncells", [20, 80, 100])
@pytest.mark.parametrize("k", [1.0, 25.0])
def test_every_derivative_matches_differences(ncells, k):
    from bempp.autograd import energy_and_gradient

    pts, cells = surface(ncells)
    rng = np.random.default_rng(ncells)
    lam, mu = (rng.standard_normal(ncells) + 1j * rng.standard_normal(ncells) for _ in range(2))
    j, dk, grad = energy_and_gradient(pts, cells, k, lam, mu)
    assert abs(j.item() - forward(pts, cells, k, lam, mu)) <= 1e-12 * np.abs(lam).sum()
    h, fd = 1e-6, np.zeros(pts.size)
    for c in range(pts.size):
        v = []
        for s in (h, -h):
            q = pts.copy().ravel()
            q[c] += s
            v.append(forward(q.reshape(-1, 3), cells, k, lam, mu))
        fd[c] = (v[0] - v[1]) / (2 * h)
    g = grad.cpu().numpy().ravel()
    assert np.abs(fd - g).max() <= 1e-6 * np.abs(g).max()
    fdk = (forward(pts, cells, k + h, lam, mu) - forward(pts, cells, k - h, lam, mu)) / (2 * h)
    assert abs(fdk - dk.item()) <= 1e-6 * max(abs(fdk), 1.0)
