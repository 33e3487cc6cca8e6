"""The work this package is used for, as timed cases through its public entry points.

Five kinds of call, each from the smallest size a program uses to the largest:

* ``device``: ``BoundaryAssembler.assemble_into_device``, the matrix left in HBM for a
  solver on the GPU;
* ``host``: ``BoundaryAssembler.assemble``, the reference's own call, into a numpy array;
* ``potential``: ``PotentialAssembler.assemble_into_device`` at points off the surface;
* ``gradient``: ``HelmholtzSingleLayerEnergy`` forward and backward (shape and wavenumber
  derivatives), on vertex positions that change from call to call;
* ``sweep``: ``helmholtz_single_layer_sweep`` over several meshes and wavenumbers.

Meshes are refined icosahedra (80, 320, .., 20,480 cells; a size between two levels is an
open surface: the first cells of the finer one) with seeded radial perturbations, so every
seed is another geometry.  ``exact`` evaluates the same quadrature sums in FP64 with plain
torch, pair by pair of quadrature points.
"""

from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bempp-rs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from bempp import shapes  # noqa: E402


def _case(name, path, kernel="laplace", op="single_layer", test="dp0", trial="", cells=0,
          cells2=0, q=6, k=0.0, precision="fp64", single=False, points=0, wavenumbers=0):
    c = dict(path=path, kernel=kernel, op=op, test=test, trial=trial or test, cells=cells,
             cells2=cells2, q=q, k=k, precision=precision, single=single, points=points,
             wavenumbers=wavenumbers)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest useful call: a first matrix with the default options (37-point rule),
        # where launches and half-empty waves count
        _case("sl_dp0_80_default", "device", cells=80, q=37),
        # a coarse model through the reference's call: numpy in, numpy out
        _case("host_sl_dp0_1280", "host", cells=1280),
        # an ordinary mesh with the options left at their defaults (37-point rule)
        _case("dl_p1_2048_default", "device", op="double_layer", test="p1", cells=2048, q=37),
        # the headline operators at full size: Laplace double layer and hypersingular, P1
        _case("dl_p1_20480", "device", op="double_layer", test="p1", cells=20480),
        _case("hs_p1_20480", "device", op="hypersingular", test="p1", cells=20480),
        # the largest matrix: Helmholtz single layer, 20,480^2 complex128
        _case("helm_sl_dp0_20480", "device", kernel="helmholtz", cells=20480, k=8.0),
        # a scattering model on a mesh that is coarse for its wavenumber (eight cells per
        # wavelength): phases that vary within a cell pair
        _case("helm_hs_p1_1280_k10", "device", kernel="helmholtz", op="hypersingular", test="p1",
              cells=1280, k=10.0),
        # the same kind of model, finer, in mixed precision
        _case("helm_dl_p1_5120_mixed", "device", kernel="helmholtz", op="double_layer", test="p1",
              cells=5120, k=5.0, precision="mixed"),
        # coupling of two bodies: open surfaces of odd sizes, different spaces, FP32 output
        _case("adl_p1_dp0_two_bodies", "device", op="adjoint_double_layer", test="p1",
              trial="dp0", cells=3001, cells2=1777, single=True),
        # field evaluation: Helmholtz double-layer potential of a P1 density
        _case("potential_helm_dl_p1", "potential", kernel="helmholtz", op="double_layer",
              test="p1", cells=5120, points=2000, k=5.0),
        # one step of a shape optimisation: energy, and its gradient by the adjoint
        _case("gradient_helm_sl_5120", "gradient", kernel="helmholtz", cells=5120, k=5.0),
        # a frequency sweep over three meshes of uneven size
        _case("sweep_3_meshes_8_k", "sweep", kernel="helmholtz", cells=5120, wavenumbers=8,
              k=20.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any operator, spaces, rule, precision and size."""
    path = rng.choice(["device"] * 7 + ["host", "potential", "gradient", "sweep"])
    if path == "sweep":
        return _case("", path, kernel="helmholtz", cells=_log_int(rng, 300, 5120),
                     wavenumbers=rng.randint(2, 12), k=round(rng.uniform(4.0, 20.0), 2))
    if path == "gradient":
        return _case("", path, kernel="helmholtz", cells=_log_int(rng, 80, 5120),
                     k=round(rng.uniform(1.0, 10.0), 2))
    kernel = rng.choice(["laplace", "helmholtz"])
    k = round(rng.uniform(1.0, 12.0), 2) if kernel == "helmholtz" else 0.0
    space = rng.choice(["dp0", "p1"])
    if path == "potential":
        return _case("", path, kernel=kernel, op=rng.choice(["single_layer", "double_layer"]),
                     test=space, cells=_log_int(rng, 80, 8000), points=_log_int(rng, 50, 3000),
                     q=rng.choice([6, 16]), k=k)
    op = rng.choice(["single_layer", "double_layer", "adjoint_double_layer", "hypersingular"])
    if op == "hypersingular":
        space = "p1"
    q = rng.choice([6, 6, 6, 16, 37])
    top = {6: 20480, 16: 6000, 37: 2500}[q]
    if path == "host":
        top = min(top, 5120)
    elif kernel == "helmholtz" and op != "single_layer":
        top = min(top, 10000)  # no dearer than the largest listed matrix
    two = rng.random() < 0.25
    cells = _log_int(rng, 80, min(top, 5120) if two else top)
    other = _log_int(rng, 80, min(top, 5120)) if two else 0
    trial = space if not two or op == "hypersingular" else rng.choice(["dp0", "p1"])
    return _case("", path, kernel=kernel, op=op, test=space, trial=trial, cells=cells,
                 cells2=other, q=q, k=k, precision=rng.choice(["fp64", "fp64", "mixed"]),
                 single=rng.random() < 0.2)


# ------------------------------------------------------------------------- inputs ---
@functools.lru_cache(maxsize=None)
def _base_mesh(ncells):
    if ncells == 2048:  # the refined octahedron of that size, whole
        return shapes.regular_sphere(4)
    level = 0
    while 20 * 4 ** level < ncells:
        level += 1
    points, cells = shapes.icosphere(level)
    cells = cells[:ncells]
    used, inverse = np.unique(cells, return_inverse=True)
    if len(used) < len(points):
        points, cells = points[used], inverse.reshape(cells.shape).astype(np.int64)
    return points, cells


def _mesh(ncells, seed):
    points, cells = _base_mesh(ncells)
    return shapes.radial_perturbation(points, seed), cells


def _meshes(case, seed):
    """(test points, test cells, trial points, trial cells or None for one mesh)."""
    points, cells = _mesh(case["cells"], 1000 * seed + 1)
    if not case["cells2"]:
        return points, cells, None, None
    p2, c2 = _mesh(case["cells2"], 1000 * seed + 2)
    return points, cells, p2 * 0.8 + np.array([2.3, 0.2, -0.1]), c2


def _sweep_meshes(case, seed):
    sizes = [max(20, case["cells"] // 16), max(20, case["cells"] // 4), case["cells"]]
    out = []
    for i, n in enumerate(sizes):
        points, cells = _base_mesh(n)
        out.append((shapes.ellipsoidal_stretch(points, 1000 * seed + 3 + i), cells))
    return out


def _wavenumbers(case, seed):
    rng = np.random.default_rng(1000 * seed + 7)
    return np.sort(rng.uniform(1.0, case["k"], case["wavenumbers"]))


def _potential_points(case, seed):
    rng = np.random.default_rng(1000 * seed + 4)
    x = rng.standard_normal((case["points"], 3))
    x *= (rng.uniform(1.3, 4.0, case["points"]) / np.linalg.norm(x, axis=1))[:, None]
    return x


def _densities(case, seed):
    rng = np.random.default_rng(1000 * seed + 5)
    v = rng.standard_normal((4, case["cells"])) / case["cells"]
    return v[0] + 1j * v[1], v[2] + 1j * v[3]


def _dtype(case):
    if case["kernel"] == "helmholtz":
        return (np.complex64, torch.complex64) if case["single"] else (np.complex128, torch.complex128)
    return (np.float32, torch.float32) if case["single"] else (np.float64, torch.float64)


def prepare(case, seed):
    from bempp.assembly.boundary import (BoundaryAssemblerOptions, OperatorType, Precision,
                                         create_helmholtz_assembler, create_laplace_assembler)
    from bempp.assembly.potential import (create_helmholtz_potential_assembler,
                                          create_laplace_potential_assembler)
    from bempp.function_space import function_space
    from ndelement.ciarlet import Continuity, Family, create_family
    from ndelement.reference_cell import ReferenceCellType
    from ndgrid.grid import Grid

    state = {"path": case["path"]}
    if case["path"] == "gradient":
        points, cells, _, _ = _meshes(case, seed)
        lam, mu = _densities(case, seed)
        state["points"] = torch.tensor(points, device="cuda", requires_grad=True)
        state["k"] = torch.tensor(case["k"], dtype=torch.float64, requires_grad=True)
        state["lam"] = torch.tensor(lam, device="cuda")
        state["mu"] = torch.tensor(mu, device="cuda")
        state["cells"] = cells
        return state
    if case["path"] == "sweep":
        state["grids"] = [Grid(p, c) for p, c in _sweep_meshes(case, seed)]
        state["ks"] = _wavenumbers(case, seed)
        state["outs"] = [torch.empty((len(state["ks"]), len(g.cells), len(g.cells)),
                                     dtype=torch.complex64, device="cuda")
                         for g in state["grids"]]
        return state
    real = np.float32 if case["single"] else np.float64
    families = {"dp0": create_family(Family.Lagrange, 0, Continuity.Discontinuous, real),
                "p1": create_family(Family.Lagrange, 1, Continuity.Standard, real)}
    operator = {"single_layer": OperatorType.SingleLayer, "double_layer": OperatorType.DoubleLayer,
                "adjoint_double_layer": OperatorType.AdjointDoubleLayer,
                "hypersingular": OperatorType.Hypersingular}[case["op"]]
    options = BoundaryAssemblerOptions()
    if case["q"] != options.regular_quadrature_degree(ReferenceCellType.Triangle):
        options.set_regular_quadrature_degree(ReferenceCellType.Triangle, case["q"])
    if case["precision"] == "mixed":
        options.set_precision(Precision.Mixed)
    ntype, ttype = _dtype(case)
    points, cells, points2, cells2 = _meshes(case, seed)
    grid = Grid(points, cells)
    space = function_space(grid, families[case["test"]])
    if case["path"] == "potential":
        create = (create_helmholtz_potential_assembler if case["kernel"] == "helmholtz"
                  else create_laplace_potential_assembler)
        args = (operator, case["k"]) if case["kernel"] == "helmholtz" else (operator,)
        state.update(assembler=create(*args, options, ntype), space=space,
                     points=torch.tensor(_potential_points(case, seed), device="cuda"))
        state["out"] = torch.empty((space.global_size, case["points"]), dtype=ttype, device="cuda")
        return state
    if case["kernel"] == "helmholtz":
        state["assembler"] = create_helmholtz_assembler(operator, case["k"], options, ntype)
    else:
        state["assembler"] = create_laplace_assembler(operator, options, ntype)
    state["test"] = state["trial"] = space
    if points2 is not None:
        state["trial"] = function_space(Grid(points2, cells2), families[case["trial"]])
    elif case["trial"] != case["test"]:
        state["trial"] = function_space(grid, families[case["trial"]])
    if case["path"] == "device":
        state["out"] = torch.empty((state["trial"].global_size, state["test"].global_size),
                                   dtype=ttype, device="cuda")
    return state


def run(state):
    from bempp.autograd import HelmholtzSingleLayerEnergy
    from bempp.sweep import helmholtz_single_layer_sweep

    path = state["path"]
    if path == "host":
        return state["assembler"].assemble(state["trial"], state["test"])
    if path == "gradient":
        value = HelmholtzSingleLayerEnergy.apply(state["points"], state["k"], state["lam"],
                                                 state["mu"], state["cells"])
        d_points, d_k = torch.autograd.grad(value, (state["points"], state["k"]))
        return {"value": value.detach(), "d_points": d_points, "d_k": d_k}
    if path == "sweep":
        return helmholtz_single_layer_sweep(state["grids"], state["ks"], state["outs"])
    stream = torch.cuda.current_stream().cuda_stream
    if path == "potential":
        state["assembler"].assemble_into_device(state["space"], state["points"], state["out"], stream)
    else:
        state["assembler"].assemble_into_device(state["trial"], state["test"], state["out"], stream)
    return state["out"]


def _dofs(cells, space):
    """Cell DOFs, numbered on first visit, and their number."""
    if space == "dp0":
        return np.arange(len(cells))[:, None], len(cells)
    _, first, inverse = np.unique(cells, return_index=True, return_inverse=True)
    number = np.empty(len(first), dtype=np.int64)
    number[np.argsort(first)] = np.arange(len(first))
    return number[inverse.reshape(cells.shape)], len(first)


def work(case):
    """Inputs read once and the matrix written once; the operations of the regular
    quadrature (additions, multiplications and each root, sine and cosine as one), each
    kernel value formed once where both orders of a pair share it.  The pairs of cells that
    touch (about a dozen per cell) are not counted."""
    q2 = case["q"] ** 2
    helm = case["kernel"] == "helmholtz"
    nb = {"dp0": 1, "p1": 3}
    parts = 2 if helm else 1
    real = 4 if case["single"] else 8
    kernel = 9 + (8 if helm else 0) + (0 if case["op"] in ("single_layer", "hypersingular") else 4)
    if case["path"] == "sweep":
        sizes = [len(c) for _, c in _sweep_meshes(case, 0)]
        pairs = sum(n * n for n in sizes) * case["wavenumbers"]
        return {"bytes": pairs * 8.0, "flops": pairs / 2 * q2 * (kernel + 2 * parts)}
    points, cells, points2, cells2 = _meshes(case, 0)
    n = len(cells)
    if case["path"] == "gradient":
        # kernel value and gradient, each pair once, then both cells' vertex sums
        return {"bytes": 24.0 * (2 * len(points) + n) + 32.0 * n,
                "flops": n * n / 2.0 * q2 * (kernel + 6 + 12)}
    ndt = _dofs(cells, case["test"])[1]
    if case["path"] == "potential":
        evals = case["points"] * n * case["q"]
        return {"bytes": float(case["points"] * ndt * parts * real + 24 * (case["points"] + len(points)) + 12 * n),
                "flops": float(evals * (kernel + 2 * parts * nb[case["test"]]))}
    same = cells2 is None
    m = n if same else len(cells2)
    nds = ndt if same and case["trial"] == case["test"] else _dofs(cells if same else cells2, case["trial"])[1]
    evals = n * m * q2 * (0.5 if same and case["trial"] == case["test"] else 1.0)
    if case["op"] == "hypersingular" and not helm:
        sums = n * m * q2 * (0.5 if same else 1.0)  # one sum per pair
    else:
        half = 0.5 if same and case["trial"] == case["test"] and case["op"] in ("single_layer", "hypersingular") else 1.0
        sums = 2.0 * half * parts * n * m * (q2 * nb[case["trial"]]
                                             + case["q"] * nb[case["test"]] * nb[case["trial"]])
    return {"bytes": float(ndt * nds * parts * real + 24 * len(points) + 12 * (n + m)),
            "flops": float(evals * kernel + sums)}


# -------------------------------------------------------------------------- exact ---
# symmetric triangle rules: orbits (first barycentric coordinates, weight)
_ORBITS = {
    6: [(0.4459484909159649, 0.4459484909159649, 0.11169079483900572),
        (0.09157621350977072, 0.09157621350977072, 0.054975871827660935)],
    16: [(1 / 3, 1 / 3, 0.07215780383889357),
         (0.17056930775176024, 0.17056930775176024, 0.05160868526735912),
         (0.4592925882927232, 0.4592925882927232, 0.047545817133642324),
         (0.05054722831703099, 0.05054722831703099, 0.016229248811599036),
         (0.7284923929554042, 0.008394777409957643, 0.013615157087217507)],
    37: [(1 / 3, 1 / 3, 0.033980018293415806),
         (0.02150968110884315, 0.02150968110884315, 0.003026168551769585),
         (0.48907694645253935, 0.48907694645253935, 0.01199720096444736),
         (0.4269414142598004, 0.4269414142598004, 0.027800983765226675),
         (0.22137228629183292, 0.22137228629183292, 0.029139242559599987),
         (0.8647077702954428, 0.1109220428034634, 0.0074827005525828355),
         (0.6235459955536756, 0.06801224355420665, 0.01732063807042419),
         (0.7223577931241879, 0.2725158177734297, 0.00479534050177163),
         (0.08789548303219734, 0.7485071158999522, 0.012089519905796903)],
}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _rule(q):
    pts, w = [], []
    for a, b, wt in _ORBITS[q]:
        c = 1.0 - a - b
        orbit = {(a, b), (b, a), (a, c), (c, a), (b, c), (c, b)}
        if abs(a - b) < 1e-15:
            orbit = {(a, a)} if abs(a - c) < 1e-12 else {(a, a), (a, c), (c, a)}
        for p in sorted(orbit):
            pts.append(p)
            w.append(wt)
    assert len(pts) == q
    dev = _device()
    return (torch.tensor(pts, dtype=torch.float64, device=dev),
            torch.tensor(w, dtype=torch.float64, device=dev))


def _basis(xi, space):
    if space == "dp0":
        return torch.ones(len(xi), 1, dtype=torch.float64, device=xi.device)
    return torch.stack([1 - xi[:, 0] - xi[:, 1], xi[:, 0], xi[:, 1]], dim=1)


class _Geometry:
    """Flat triangles: v0, t0, t1, Jacobian determinant, unit normal."""

    def __init__(self, points, cells):
        v = points[cells]
        self.v0, self.t0, self.t1 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        cross = torch.linalg.cross(self.t0, self.t1)
        self.jdet = torch.linalg.vector_norm(cross, dim=1)
        self.normal = cross / self.jdet[:, None]

    def at(self, xi, cells=None):
        v0, t0, t1 = (a if cells is None else a[cells] for a in (self.v0, self.t0, self.t1))
        return v0[:, None] + xi[None, :, :1] * t0[:, None] + xi[None, :, 1:] * t1[:, None]

    def curls(self, cells, space):
        t0, t1 = self.t0[cells], self.t1[cells]
        if space == "dp0":
            return torch.zeros_like(t0)[:, None]
        return torch.stack([t0 - t1, t1, -t0], dim=1)


def _adjacent_pairs(cells):
    """Ordered pairs of cells that share a vertex, with the reference's rule of each."""
    n = len(cells)
    order = np.argsort(cells.ravel(), kind="stable")
    owner, vertex = order // 3, cells.ravel()[order]
    start = np.searchsorted(vertex, vertex, side="left")
    count = np.searchsorted(vertex, vertex, side="right") - start
    left = np.repeat(owner, count)
    offset = np.arange(len(left)) - np.repeat(np.cumsum(count) - count, count)
    pairs = np.unique(left * n + owner[np.repeat(start, count) + offset])
    test, trial = pairs // n, pairs % n
    same = cells[test][:, :, None] == cells[trial][:, None, :]
    groups = {}
    shared = same.sum(axis=(1, 2))
    key = (same.reshape(len(test), 9) * (1 << np.arange(9))).sum(axis=1)
    for value in np.unique(key):
        at = np.nonzero(key == value)[0]
        m = same[at[0]]
        if shared[at[0]] == 3:
            tp = sp = [0, 1, 2]
        else:
            sp = [j for j in range(3) if m[:, j].any()]  # ascending in the trial cell
            tp = [int(np.nonzero(m[:, j])[0][0]) for j in sp]
            if len(sp) == 2 and tp[0] < tp[1] and sp[0] > sp[1]:
                tp, sp = tp[::-1], sp[::-1]
            tp = tp + [i for i in range(3) if i not in tp]
            sp = sp + [j for j in range(3) if j not in sp]
        groups[int(value)] = (test[at], trial[at], int(shared[at[0]]), tp, sp)
    return list(groups.values())


def _duffy(shared, tp, sp, order=4):
    """Sauter-Schwab rules (section 5.2) on {0 <= x2 <= x1 <= 1}^2: identical, common edge,
    common vertex; n Gauss-Legendre points on each coordinate of the 4-cube."""
    x, w = np.polynomial.legendre.leggauss(order)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    z, a, b, c = (g.ravel() for g in np.meshgrid(x, x, x, x, indexing="ij"))
    wt = np.prod([g.ravel() for g in np.meshgrid(w, w, w, w, indexing="ij")], axis=0)
    j0 = z ** 3 * a ** 2
    if shared == 3:
        regions = [(z, z * (1 - a + a * b), z * (1 - a * b * c), z * (1 - a), j0 * b),
                   (z * (1 - a * b * c), z * (1 - a), z, z * (1 - a + a * b), j0 * b),
                   (z, z * a * (1 - b + b * c), z * (1 - a * b), z * a * (1 - b), j0 * b),
                   (z * (1 - a * b), z * a * (1 - b), z, z * a * (1 - b + b * c), j0 * b),
                   (z * (1 - a * b * c), z * a * (1 - b * c), z, z * a * (1 - b), j0 * b),
                   (z, z * a * (1 - b), z * (1 - a * b * c), z * a * (1 - b * c), j0 * b)]
    elif shared == 2:
        regions = [(z, z * a * c, z * (1 - a * b), z * a * (1 - b), j0),
                   (z, z * a, z * (1 - a * b * c), z * a * b * (1 - c), j0 * b),
                   (z * (1 - a * b), z * a * (1 - b), z, z * a * b * c, j0 * b),
                   (z * (1 - a * b * c), z * a * b * (1 - c), z, z * a, j0 * b),
                   (z * (1 - a * b * c), z * a * (1 - b * c), z, z * a * b, j0 * b)]
    else:
        regions = [(z, z * a, z * b, z * b * c, z ** 3 * b),
                   (z * b, z * b * a, z, z * c, z ** 3 * b)]

    def reference(x1, x2, perm):
        bary = (1 - x1, x1 - x2, x2)
        out = np.zeros((len(x1), 2))
        for i in range(3):
            if perm[i]:
                out[:, perm[i] - 1] += bary[i]
        return out

    dev = _device()
    xi = np.concatenate([reference(r[0], r[1], tp) for r in regions])
    eta = np.concatenate([reference(r[2], r[3], sp) for r in regions])
    wts = np.concatenate([wt * r[4] for r in regions])
    return tuple(torch.tensor(v, dtype=torch.float64, device=dev) for v in (xi, eta, wts))


def _kernel(d, k, kind, op, nx, ny):
    """Kernel values of differences d = x - y (..., 3); real and imaginary parts."""
    r = torch.sqrt((d * d).sum(-1))
    g = 1.0 / (4.0 * math.pi * r)
    if op in ("single_layer", "hypersingular"):
        if kind == "laplace":
            return g, None
        return g * torch.cos(k * r), g * torch.sin(k * r)
    dn = (d * ny).sum(-1) if op == "double_layer" else -(d * nx).sum(-1)
    f = g * dn / (r * r)
    if kind == "laplace":
        return f, None
    cos, sin = torch.cos(k * r), torch.sin(k * r)
    return f * (cos + k * r * sin), f * (sin - k * r * cos)


def _pair_blocks(parts, w, phi, psi, gx, gy, tc, sc, kind, op, k, test, trial):
    """Local blocks from the kernel values of tensor rules (..., npts) with weights w and
    basis values phi, psi at the points: sum over the points, times the Jacobians."""
    jj = gx.jdet[tc] * gy.jdet[sc]
    out = []
    for part in parts:
        block = torch.einsum("np,p,pa,pb->nab", part, w, phi, psi) if op != "hypersingular" or kind == "helmholtz" else None
        if op == "hypersingular":
            cc = torch.einsum("nad,nbd->nab", gx.curls(tc, test), gy.curls(sc, trial))
            total = (part * w).sum(1)[:, None, None] * cc
            if kind == "helmholtz":
                nn = (gx.normal[tc] * gy.normal[sc]).sum(1) * jj
                total = total - (k * k * nn)[:, None, None] * block
            out.append(total)
        else:
            out.append(block * jj[:, None, None])
    return out


def _assemble(points, cells, points2, cells2, kind, op, k, test, trial, q, dev):
    """The matrix (real and imaginary parts) as (trial DOFs, test DOFs) tensors."""
    same = points2 is None
    P = torch.as_tensor(points, dtype=torch.float64, device=dev)
    C = torch.as_tensor(cells, device=dev)
    gx = _Geometry(P, C)
    gy = gx if same else _Geometry(torch.as_tensor(points2, dtype=torch.float64, device=dev),
                                   torch.as_tensor(cells2, device=dev))
    tcells = cells if same else cells2
    (td, nt), (sd, ns) = _dofs(cells, test), _dofs(tcells, trial)
    td, sd = torch.as_tensor(td, device=dev), torch.as_tensor(sd, device=dev)
    parts = 2 if kind == "helmholtz" else 1
    mats = [torch.zeros(ns, nt, dtype=torch.float64, device=dev) for _ in range(parts)]
    xi, w = _rule(q)
    phi, psi = _basis(xi, test), _basis(xi, trial)
    Y = gy.at(xi)
    n, m = len(cells), len(tcells)
    groups = _adjacent_pairs(cells) if same else []
    touch = None
    if same:
        pt = np.concatenate([g[0] for g in groups])
        ps = np.concatenate([g[1] for g in groups])
        by = np.argsort(pt, kind="stable")
        touch = (pt[by], ps[by])
    budget = 24_000_000 if dev.type == "cuda" else 2_000_000
    step = max(1, budget // (m * q * q))
    cols = max(1, min(m, budget // (q * q)))
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        X = gx.at(xi, torch.arange(i0, i1, device=dev))
        for j0 in range(0, m, cols):
            j1 = min(m, j0 + cols)
            d = [X[:, None, :, None, e] - Y[None, j0:j1, None, :, e] for e in range(3)]
            r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)  # (i, j, p, q)
            g = 1.0 / (4.0 * math.pi * r)
            if op in ("double_layer", "adjoint_double_layer"):
                if op == "double_layer":
                    nv = [gy.normal[None, j0:j1, None, None, e] for e in range(3)]
                    dn = d[0] * nv[0] + d[1] * nv[1] + d[2] * nv[2]
                else:
                    nv = [gx.normal[i0:i1, None, None, None, e] for e in range(3)]
                    dn = -(d[0] * nv[0] + d[1] * nv[1] + d[2] * nv[2])
                g = g * dn / (r * r)
            if kind == "laplace":
                vals = [g]
            else:
                cos, sin = torch.cos(k * r), torch.sin(k * r)
                if op in ("double_layer", "adjoint_double_layer"):
                    vals = [g * (cos + k * r * sin), g * (sin - k * r * cos)]
                else:
                    vals = [g * cos, g * sin]
            jj = gx.jdet[i0:i1, None] * gy.jdet[None, j0:j1]
            skip = None
            if touch is not None:
                lo, hi = np.searchsorted(touch[0], [i0, i1])
                a, b = touch[0][lo:hi] - i0, touch[1][lo:hi]
                inside = (b >= j0) & (b < j1)
                skip = (torch.as_tensor(a[inside], device=dev), torch.as_tensor(b[inside] - j0, device=dev))
            for part, v in enumerate(vals):
                if op == "hypersingular":
                    cc = torch.einsum("iad,jbd->ijab", gx.curls(torch.arange(i0, i1, device=dev), test),
                                      gy.curls(torch.arange(j0, j1, device=dev), trial))
                    block = torch.einsum("ijpq,p,q->ij", v, w, w)[..., None, None] * cc
                    if kind == "helmholtz":
                        nn = (gx.normal[i0:i1] @ gy.normal[j0:j1].T) * jj
                        block = block - (k * k * nn)[..., None, None] * torch.einsum(
                            "ijpq,pa,qb->ijab", v, phi * w[:, None], psi * w[:, None])
                else:
                    block = torch.einsum("ijpq,pa,qb->ijab", v, phi * w[:, None], psi * w[:, None])
                    block = block * jj[..., None, None]
                if skip is not None:
                    block[skip[0], skip[1]] = 0.0
                rows = td[i0:i1].reshape(-1)
                flat = block.permute(1, 3, 0, 2).reshape((j1 - j0) * psi.shape[1], (i1 - i0) * phi.shape[1])
                if test == "dp0" and trial == "dp0":
                    mats[part][j0:j1, i0:i1] += flat
                else:
                    wide = torch.zeros(ns, flat.shape[1], dtype=torch.float64, device=dev)
                    wide.index_add_(0, sd[j0:j1].reshape(-1), flat)
                    mats[part].index_add_(1, rows, wide)
    for tc_all, sc_all, shared, tp, sp in groups:
        xs, es, ws = _duffy(shared, tp, sp)
        fx, fy = _basis(xs, test), _basis(es, trial)
        most = max(1, budget // len(ws))
        for s in range(0, len(tc_all), most):
            tc = torch.as_tensor(tc_all[s:s + most], device=dev)
            sc = torch.as_tensor(sc_all[s:s + most], device=dev)
            d = gx.at(xs, tc) - gy.at(es, sc)
            vals = _kernel(d, k, kind, op, gx.normal[tc][:, None], gy.normal[sc][:, None])
            blocks = _pair_blocks([v for v in vals if v is not None], ws, fx, fy, gx, gy, tc, sc,
                                  kind, op, k, test, trial)
            at = (sd[sc][:, None, :] * nt + td[tc][:, :, None]).reshape(-1)
            for part, block in enumerate(blocks):
                mats[part].view(-1).index_add_(0, at, block.reshape(-1))
    return mats


def _complete(mats):
    return mats[0] if len(mats) == 1 else torch.complex(mats[0], mats[1])


def _energy(points, k, lam, mu, cells, dev):
    """Value, d/dpoints and d/dk by automatic differentiation of the sums."""
    C = torch.as_tensor(cells, device=dev)
    P = torch.tensor(points, dtype=torch.float64, device=dev, requires_grad=True)
    K = torch.tensor(k, dtype=torch.float64, device=dev, requires_grad=True)
    L, M = (torch.as_tensor(v, device=dev) for v in (lam, mu))
    xi, w = _rule(6)
    groups = _adjacent_pairs(cells)
    pt = np.concatenate([g[0] for g in groups])
    ps = np.concatenate([g[1] for g in groups])
    by = np.argsort(pt, kind="stable")
    pt, ps = pt[by], ps[by]
    n, q = len(cells), len(w)
    total, dp, dk = 0.0, torch.zeros_like(P), torch.zeros_like(K)

    def add(value):
        nonlocal total, dp, dk
        a, b = torch.autograd.grad(value, (P, K))
        total, dp, dk = total + float(value.detach()), dp + a, dk + b

    step = max(1, (8_000_000 if dev.type == "cuda" else 1_000_000) // (n * q * q))
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        g = _Geometry(P, C)
        c = torch.conj(L[i0:i1])[:, None] * M[None, :]
        lo, hi = np.searchsorted(pt, [i0, i1])
        c[torch.as_tensor(pt[lo:hi] - i0, device=dev), torch.as_tensor(ps[lo:hi], device=dev)] = 0.0
        X, Y = g.at(xi, torch.arange(i0, i1, device=dev)), g.at(xi)
        keep = (c != 0)[:, :, None, None]
        r2 = sum((X[:, None, :, None, e] - Y[None, :, None, :, e]) ** 2 for e in range(3))
        r = torch.sqrt(torch.where(keep, r2, torch.ones_like(r2)))
        f = torch.einsum("ijpq,p,q->ij", (c.real[:, :, None, None] * torch.cos(K * r)
                                          - c.imag[:, :, None, None] * torch.sin(K * r)) / r, w, w)
        add((f * g.jdet[i0:i1, None] * g.jdet[None, :]).sum() / (4 * math.pi))
    for tc_all, sc_all, shared, tp, sp in groups:
        xs, es, ws = _duffy(shared, tp, sp)
        most = max(1, 4_000_000 // len(ws))
        for s in range(0, len(tc_all), most):
            tc = torch.as_tensor(tc_all[s:s + most], device=dev)
            sc = torch.as_tensor(sc_all[s:s + most], device=dev)
            g = _Geometry(P, C)
            r = torch.sqrt(((g.at(xs, tc) - g.at(es, sc)) ** 2).sum(-1))
            c = torch.conj(L[tc]) * M[sc]
            f = ((c.real[:, None] * torch.cos(K * r) - c.imag[:, None] * torch.sin(K * r)) / r) @ ws
            add((f * g.jdet[tc] * g.jdet[sc]).sum() / (4 * math.pi))
    return {"value": torch.tensor(total, dtype=torch.float64), "d_points": dp, "d_k": dk}


def exact(case, seed):
    dev = _device()
    evals = float(case["cells"]) * (case["cells2"] or case["cells"]) * case["q"] ** 2
    if dev.type == "cpu" and evals > 3e8:
        return None
    if case["path"] == "gradient":
        points, cells, _, _ = _meshes(case, seed)
        return _energy(points, case["k"], *_densities(case, seed), cells, dev)
    if case["path"] == "sweep":
        return [torch.stack([_complete(_assemble(p, c, None, None, "helmholtz", "single_layer", float(k),
                                                 "dp0", "dp0", 6, dev))
                             for k in _wavenumbers(case, seed)])
                for p, c in _sweep_meshes(case, seed)]
    points, cells, points2, cells2 = _meshes(case, seed)
    if case["path"] == "potential":
        X = torch.as_tensor(_potential_points(case, seed), device=dev)
        g = _Geometry(torch.as_tensor(points, dtype=torch.float64, device=dev),
                      torch.as_tensor(cells, device=dev))
        xi, w = _rule(case["q"])
        psi = _basis(xi, case["test"]) * w[:, None]
        dofs, nd = _dofs(cells, case["test"])
        dofs = torch.as_tensor(dofs, device=dev)
        Y = g.at(xi)
        parts = 2 if case["kernel"] == "helmholtz" else 1
        mats = [torch.zeros(nd, len(X), dtype=torch.float64, device=dev) for _ in range(parts)]
        step = max(1, 8_000_000 // (len(X) * case["q"]))
        for j0 in range(0, len(cells), step):
            y = Y[j0:j0 + step]
            d = X[None, None] - y[:, :, None]
            vals = _kernel(d, case["k"], case["kernel"], case["op"], None,
                           g.normal[j0:j0 + step, None, None])
            for part in range(parts):
                block = torch.einsum("jqi,qb,j->jbi", vals[part], psi, g.jdet[j0:j0 + step])
                mats[part].index_add_(0, dofs[j0:j0 + step].reshape(-1), block.reshape(-1, len(X)))
        return _complete(mats)
    mat = _complete(_assemble(points, cells, points2, cells2, case["kernel"], case["op"], case["k"],
                              case["test"], case["trial"], case["q"], dev))
    # assemble() returns the test x trial matrix, column by column; the device call its transpose
    return mat.T.cpu().numpy() if case["path"] == "host" else mat
