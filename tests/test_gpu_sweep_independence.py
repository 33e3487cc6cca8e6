"""Wavenumbers that share a pass of the sweep do not change one another's matrices: k = 1 beside
wavenumbers up to 1e5 (phases of thousands per cell) and beside infinite and NaN ones."""

import numpy as np
import pytest

from bempp import shapes
from ndgrid.grid import Grid

pytestmark = pytest.mark.gpu


def sweep(ks):
    import torch

    from bempp.sweep import helmholtz_single_layer_sweep, set_tuning

    points, cells = shapes.icosphere(2)
    grid = Grid(points * 2.0, cells)  # radii of about 0.3: k (rad + rad) up to 6e4
    out = torch.full((len(ks), len(cells), len(cells)), float("nan"), dtype=torch.complex64, device="cuda")
    set_tuning(8, 4, 1)  # all wavenumbers in one pass
    try:
        helmholtz_single_layer_sweep([grid], np.array(ks), [out])
    finally:
        set_tuning()
    return out.cpu().numpy()


@pytest.mark.parametrize("others", [[100.0], [1e4], [1e5], [1e3, 1e4, 1e5], [30.0, 1e6, 3e4],
                                    [float("nan")], [float("inf")], [2.0, float("inf"), float("nan")]])
def test_one_wavenumber_beside_others(others):
    """Tolerance: the far pairs are FP32 sums of 36 terms in either grouping, as in the other
    sweep tests."""
    alone = sweep([1.0])[0]
    together = sweep([1.0] + others)
    assert np.abs(together[0] - alone).max() <= 1e-6 * np.abs(alone).max()
    for k, a in zip(others, together[1:]):
        if np.isfinite(k):
            assert np.isfinite(a).all()
        else:
            assert not np.isfinite(a).any()
