"""Cells that nearly touch without sharing a vertex, against the oracle: two parallel sheets in
one grid, turned so that no coordinate is exact, at gaps of 1e-2 to 1e-8 of a cell's edge, the
rule points of facing cells opposite each other (equal sheets) or not (a coarse and a fine one).

Tolerance: both sides form rule points with errors of a few eps |x|, so 1/r of facing points is
off by up to 8 eps |x| / gap, 1/r^3 by three times that and the normal factor (x - y).n once
more: 64 eps |x| / gap beside the parity tests' bound."""

import numpy as np
import pytest

from bempp.assembly.boundary import BoundaryAssemblerOptions
from bempp.assembly.potential import (create_helmholtz_potential_assembler,
                                      create_laplace_potential_assembler)
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndelement.reference_cell import ReferenceCellType
from ndgrid.grid import Grid
from oracle import oracle, potential

from test_gpu_parity import FP64_TOL, OPS, SPACES, gpu_assemble, oracle_assemble, rel_err

pytestmark = pytest.mark.gpu

GAPS = [1e-2, 1e-4, 1e-6, 1e-8]


def sheet(n):
    x = np.linspace(0.0, 1.0, n + 1)
    points = np.stack([np.repeat(x, n + 1), np.tile(x, n + 1), np.zeros((n + 1) ** 2)], axis=1)
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]).ravel()
    cells = np.stack([a, a + n + 1, a + 1, a + n + 1, a + n + 2, a + 1], axis=1).reshape(-1, 3)
    return points, cells


def turned(points):
    q, _ = np.linalg.qr(np.random.default_rng(7).standard_normal((3, 3)))
    return points @ q.T + np.array([0.1, -0.2, 0.3])


def sheets(gap, n1=3, n2=3):
    """Two sheets, `gap` edges (1 / n1) apart, and the tolerance."""
    (p1, c1), (p2, c2) = sheet(n1), sheet(n2)
    p2 = p2 + np.array([0.0, 0.0, gap / n1])
    points = turned(np.vstack([p1, p2]))
    size = np.abs(points).max()
    tol = FP64_TOL + 64 * np.finfo(float).eps * size * n1 / gap
    return Grid(points, np.vstack([c1, c2 + len(p1)])), tol


@pytest.mark.parametrize("gap", GAPS)
@pytest.mark.parametrize("q", [6, 16])
@pytest.mark.parametrize("kernel,op,k,sp", [("laplace", "single_layer", 0.0, "dp0"),
                                            ("laplace", "double_layer", 0.0, "p1"),
                                            ("laplace", "adjoint_double_layer", 0.0, "dp1"),
                                            ("laplace", "hypersingular", 0.0, "p1"),
                                            ("helmholtz", "single_layer", 0.5, "dp0"),
                                            ("helmholtz", "double_layer", 1.5, "p1"),
                                            ("helmholtz", "adjoint_double_layer", 20.0, "p1"),
                                            ("helmholtz", "hypersingular", 20.0, "p1")])
def test_facing_sheets(gap, q, kernel, op, k, sp):
    grid, tol = sheets(gap)
    a = gpu_assemble(grid, kernel, op, k, SPACES[sp], q=q, one_space=True)
    assert rel_err(a, oracle_assemble(grid, kernel, op, k, SPACES[sp], SPACES[sp], q=q)) <= tol


@pytest.mark.parametrize("gap", GAPS)
@pytest.mark.parametrize("kernel,op,k,test,trial", [("laplace", "single_layer", 0.0, "p1", "dp0"),
                                                    ("laplace", "adjoint_double_layer", 0.0, "dp0", "p1"),
                                                    ("helmholtz", "double_layer", 3.0, "dp0", "p1")])
def test_coarse_against_fine_sheet(gap, kernel, op, k, test, trial):
    grid, tol = sheets(gap, 1, 5)
    a = gpu_assemble(grid, kernel, op, k, SPACES[test], SPACES[trial], q=37)
    assert rel_err(a, oracle_assemble(grid, kernel, op, k, SPACES[test], SPACES[trial], q=37)) <= tol


@pytest.mark.parametrize("gap", GAPS)
@pytest.mark.parametrize("q", [6, 16])
@pytest.mark.parametrize("kernel,op,k,degree", [("laplace", "single_layer", 0.0, 0),
                                                ("laplace", "double_layer", 0.0, 1),
                                                ("helmholtz", "single_layer", 2.0, 2),
                                                ("helmholtz", "double_layer", 2.0, 1)])
def test_potential_above_a_sheet(gap, q, kernel, op, k, degree):
    """Points `gap` edges above the rule points of a sheet's cells."""
    n = 3
    p, c = sheet(n)
    x, _ = oracle.simplex_rule(q)
    v = p[c]
    above = (v[:, :1] + x[:, :1] * (v[:, 1:2] - v[:, :1]) + x[:, 1:] * (v[:, 2:] - v[:, :1])).reshape(-1, 3)
    above = turned(above + np.array([0.0, 0.0, gap / n]))
    points = turned(p)
    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, q)
    a = (create_laplace_potential_assembler(OPS[op], opts) if kernel == "laplace"
         else create_helmholtz_potential_assembler(OPS[op], k, opts))
    space = function_space(Grid(points, c), create_family(
        Family.Lagrange, degree, Continuity.Standard if degree else Continuity.Discontinuous))
    o = potential.potential(above, points, c.astype(np.int64), kernel, op, k=k, degree=degree,
                            continuous=degree > 0, q_regular=q)
    tol = FP64_TOL + 64 * np.finfo(float).eps * np.abs(above).max() * n / gap
    assert rel_err(a.assemble(space, above), o) <= tol


@pytest.mark.parametrize("gap", GAPS[:3])
@pytest.mark.parametrize("k", [0.5, 20.0])
@pytest.mark.parametrize("q", [6, 16])
def test_gradient_between_sheets(gap, k, q):
    """lambda lives on one sheet and mu on the other, so that only facing pairs count.  Against
    the rule's sum differentiated by torch: grad 1/r loses as the double layer does."""
    import torch

    from bempp.autograd import energy_and_gradient

    grid, tol = sheets(gap)
    points, cells = np.array(grid.points), np.array(grid.cells, dtype=np.int64)
    n = len(cells) // 2
    rng = np.random.default_rng(3)
    lam, mu = (rng.standard_normal(2 * n) + 1j * rng.standard_normal(2 * n) for _ in range(2))
    lam[n:] = 0.0
    mu[:n] = 0.0
    j, dk, grad = energy_and_gradient(points, cells, k, lam, mu, regular_points=q)
    xi, w = oracle.simplex_rule(q)
    phi = torch.tensor(np.stack([1.0 - xi.sum(1), xi[:, 0], xi[:, 1]], axis=1))
    w = torch.tensor(w)
    p = torch.tensor(points, requires_grad=True)
    kt = torch.tensor(k, dtype=torch.float64, requires_grad=True)
    v = p[torch.tensor(cells)]
    jdet = torch.linalg.norm(torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]), dim=1)
    x = torch.einsum("qa,cad->cqd", phi, v)
    r = torch.linalg.norm(x[:n, None, :, None] - x[None, n:, None, :], dim=-1)
    a = torch.einsum("ijpq,p,q->ij", torch.polar(1.0 / r, kt * r), w.cdouble(), w.cdouble())
    a = a * jdet[:n, None] * jdet[None, n:] / (4 * np.pi)
    value = (torch.tensor(lam[:n]).conj() @ a @ torch.tensor(mu[n:])).real
    value.backward()
    assert abs(j.item() - value.item()) <= tol * max(abs(value.item()), a.abs().max().item())
    assert np.abs(grad.cpu().numpy() - p.grad.numpy()).max() <= tol * p.grad.abs().max().item()
    assert abs(dk.item() - kt.grad.item()) <= tol * max(abs(kt.grad.item()), 1.0)
