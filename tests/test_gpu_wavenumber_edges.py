"""Wavenumbers at the edges: infinite and NaN, negative, and phases around 2^51, from which on
their last digit is worth half a radian or more."""

import numpy as np
import pytest

from bempp import shapes
from bempp.assembly.boundary import Precision
from bempp.assembly.potential import create_helmholtz_potential_assembler
from bempp.function_space import function_space
from ndelement.ciarlet import Continuity, Family, create_family
from ndgrid.grid import Grid

from test_gpu_parity import OPS, SPACES, gpu_assemble

pytestmark = pytest.mark.gpu

NON_FINITE = [float("nan"), float("inf"), -float("inf")]


def sphere(level=1):
    points, cells = shapes.icosphere(level)
    return Grid(shapes.radial_perturbation(points, seed=5), cells)


@pytest.mark.parametrize("k", NON_FINITE)
@pytest.mark.parametrize("q", [6, 16])
@pytest.mark.parametrize("op,sp", [("single_layer", "dp0"), ("single_layer", "p1"),
                                   ("double_layer", "p1"), ("hypersingular", "p1")])
def test_non_finite_wavenumber_is_not_hidden(k, q, op, sp):
    """No entry is finite: a NaN phase must not read as a phase of 0."""
    a = gpu_assemble(sphere(), "helmholtz", op, k, SPACES[sp], q=q, one_space=True)
    assert not np.isfinite(a).any()


@pytest.mark.parametrize("k", NON_FINITE)
@pytest.mark.parametrize("op", ["single_layer", "double_layer"])
def test_non_finite_wavenumber_of_a_potential_and_a_gradient(k, op):
    grid = sphere()
    x = 3.0 * np.random.default_rng(0).standard_normal((5, 3))
    space = function_space(grid, create_family(Family.Lagrange, 1, Continuity.Standard))
    assert not np.isfinite(create_helmholtz_potential_assembler(OPS[op], k).assemble(space, x)).any()
    if op == "single_layer":
        from bempp.autograd import energy_and_gradient

        ones = np.ones(len(grid.cells), dtype=complex)
        j, dk, grad = energy_and_gradient(np.array(grid.points), np.array(grid.cells, dtype=np.int64),
                                          k, ones, ones)
        assert not np.isfinite(j.item()) and not np.isfinite(dk.item())
        assert not np.isfinite(grad.cpu().numpy()).any()


@pytest.mark.parametrize("exponent", [50, 51, 52, 56])
def test_huge_phases_keep_their_modulus(exponent):
    """One-point rule: every regular entry is w^2 jdet jdet e^{ikr} / (4 pi r), so |entry| is the
    Laplace entry, to a few rounding errors, whatever the phase k r of about 2^exponent is."""
    grid = sphere()
    v = np.asarray(grid.cells)
    apart = ~(v[:, None, :, None] == v[None, :, None, :]).any(axis=(2, 3))
    still = gpu_assemble(grid, "laplace", "single_layer", q=1)
    a = gpu_assemble(grid, "helmholtz", "single_layer", 2.0 ** exponent, q=1)
    assert np.abs(np.abs(a[apart]) / still[apart] - 1.0).max() <= 1e-12


@pytest.mark.parametrize("k", [1.0, 30.0, 300.0])
@pytest.mark.parametrize("precision", [Precision.FP64, Precision.Mixed])
@pytest.mark.parametrize("op,sp", [("single_layer", "dp0"), ("double_layer", "p1")])
def test_negative_wavenumber_gives_the_conjugate(k, precision, op, sp):
    """Bit for bit up to the order of the atomic sums: 1e-14 of the largest entry in FP64, FP32
    rounding in mixed precision."""
    a, b = (gpu_assemble(sphere(2), "helmholtz", op, v, SPACES[sp], precision=precision, one_space=True)
            for v in (k, -k))
    tol = 1e-14 if precision == Precision.FP64 else 1e-6
    assert np.abs(b - a.conj()).max() <= tol * np.abs(a).max()


@pytest.mark.parametrize("k", [1.0, 30.0, 300.0])
def test_negative_wavenumber_in_a_sweep(k):
    import torch

    from bempp.sweep import helmholtz_single_layer_sweep

    grid = sphere(2)
    n = len(grid.cells)
    outs = [torch.empty((1, n, n), dtype=torch.complex64, device="cuda") for _ in range(2)]
    for out, v in zip(outs, (k, -k)):
        helmholtz_single_layer_sweep([grid], np.array([v]), [out])
    d = (outs[1] - outs[0].conj()).abs().max().item()
    assert d <= 1e-6 * outs[0].abs().max().item()


@pytest.mark.parametrize("k", [1.0, 30.0, 300.0])
@pytest.mark.parametrize("q,mixed", [(6, False), (16, False), (6, True)])
def test_negative_wavenumber_of_a_gradient(k, q, mixed):
    """J(-k) with conjugated densities is J(k): the same gradient, the opposite dJ/dk."""
    from bempp.autograd import energy_and_gradient

    grid = sphere(1)
    points, cells = np.array(grid.points), np.array(grid.cells, dtype=np.int64)
    rng = np.random.default_rng(1)
    lam, mu = (rng.standard_normal(len(cells)) + 1j * rng.standard_normal(len(cells)) for _ in range(2))
    j, dk, g = energy_and_gradient(points, cells, k, lam, mu, regular_points=q, mixed=mixed)
    j2, dk2, g2 = energy_and_gradient(points, cells, -k, lam.conj(), mu.conj(), regular_points=q, mixed=mixed)
    tol = 1e-6 if mixed else 1e-12
    assert abs(j.item() - j2.item()) <= tol * max(abs(j.item()), 1.0)
    assert abs(dk.item() + dk2.item()) <= tol * max(abs(dk.item()), 1.0)
    assert (g - g2).abs().max().item() <= tol * max(g.abs().max().item(), 1.0)
