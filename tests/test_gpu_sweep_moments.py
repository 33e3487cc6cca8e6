"""Sweep at the edges of its tiles, of its passes of eight wavenumbers and of its phase ranges.

Against one FP64 assembly per wavenumber: ragged surfaces (one partial tile, tiles and a
remainder), 9 wavenumbers (one pass and one more) that mix the ranges in one pass, k = 0 among
them.  Tolerance 1e-6 of the norm and of the largest entry: complex64 rounding is 6e-8, an FP32
sum of 36 terms with FP32 distances a few times that.
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
    pts, cells = shapes.ellipsoidal_stretch(pts, ncells), np.asarray(cells)[:ncells]
    used, cells = np.unique(cells, return_inverse=True)
    return Grid(np.ascontiguousarray(pts[used]), cells.reshape(-1, 3))


@pytest.mark.parametrize("ks", [[3.0], [0.0, 2.0], [0.0, 1.0, 2.5, 4.0, 6.0, 9.0, 14.0, 30.0, 60.0],
                                [40.0, 80.0, 120.0]])
@pytest.mark.parametrize("tuning", [(1, 2, 1), (8, 4, 1), (32, 3, 2)])
def test_ranges_and_remainders(ks, tuning):
    import torch

    from bempp.sweep import helmholtz_single_layer_sweep, set_tuning

    grids = [surface(n) for n in (20, 100, 1000)]
    set_tuning(*tuning)
    try:
        outs = [torch.full((len(ks), len(g.cells), len(g.cells)), float("nan"), dtype=torch.complex64,
                           device="cuda") for g in grids]
        helmholtz_single_layer_sweep(grids, np.array(ks), outs)
    finally:
        set_tuning()
    fam = create_family(Family.Lagrange, 0, Continuity.Discontinuous)
    opts = BoundaryAssemblerOptions()
    opts.set_regular_quadrature_degree(ReferenceCellType.Triangle, 6)
    for g, o in zip(grids, outs):
        sp = function_space(g, fam)
        n = sp.global_size
        for j, k in enumerate(ks):
            ref = torch.empty((n, n), dtype=torch.complex128, device="cuda")
            a = create_helmholtz_assembler(OperatorType.SingleLayer, k, opts)
            a.assemble_into_device(sp, sp, ref, torch.cuda.current_stream().cuda_stream)
            d = o[j].to(torch.complex128) - ref
            assert (torch.linalg.norm(d) <= 1e-6 * torch.linalg.norm(ref)).item(), (n, k)
            assert d.abs().max().item() <= 1e-6 * ref.abs().max().item(), (n, k)
