"""Over-relaxed passes and the averaged-face coarse coefficients of the solves
(geometric hierarchy, cell coefficients): the converged solution equals the
FP64 oracle's at every form of the V-cycle -- odd, merged and periodic levels,
one to three sweeps on either side, high contrasts, single and batched -- and
takes no more V-cycles than the oracle's plain red-black Gauss-Seidel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver, workloads as W  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

PER, DIR, ZG = ["PERI"] * 2, ["DIRC"] * 2, ["ZGRD"] * 2


@pytest.fixture(scope="module")
def handle():
    return capi.Handle(0)


def _field(k, bc, seed=3):
    nz, ny, nx = k.shape
    g = (nz + 2, ny + 2, nx + 2)
    dc = np.ones(g)
    dc[1:-1, 1:-1, 1:-1] = k
    src = np.random.default_rng(seed).uniform(-1.0, 1.0, g)
    return Problem(nx, ny, nz, (1.0, 1.0, 1.0), dcoeff=dc, source=src, bc=bc, bcvals=[0.0] * 6)


def _layer(shape, contrast, lo, hi):
    k = np.ones(shape)
    k[lo:hi] = contrast
    return k


CASES = {
    "dirichlet_33": lambda: W.poisson_dirichlet(33),
    "dirichlet_ragged": lambda: W.poisson_dirichlet(41, ny=23, nz=30),
    "tiny": lambda: W.poisson_dirichlet(7, ny=9, nz=11),
    "plasma_33": lambda: W.plasma_poisson(33, slab_cells=2),
    "plasma_34": lambda: W.plasma_poisson(34, slab_cells=3, eps_slab=10.0),
    "odd_periodic": lambda: _field(np.random.default_rng(1).uniform(0.5, 2.0, (27, 25, 31)), PER + PER + DIR),
    "thin_layer": lambda: _field(_layer((38, 21, 20), 70.0, 12, 14), DIR + ZG + ZG),
    "checkerboard": lambda: _field(np.where(np.indices((32, 32, 32)).sum(0) % 2 == 0, 1.0, 20.0), DIR * 3),
    "reaction": lambda: W.random_operator(29, 20, 26, bc=["DIRC", "ZGRD", "PERI", "PERI", "DIRC", "FLUX"], seed=7,
                                          vel=False, reac=True, timederiv=True),
}


def _reference(p, nu1, nu2):
    mg = O.RowsMG(p, hier=O.HIER_GEOM, nu1=nu1, nu2=nu2)
    b = O.build_rhs(p)
    x, hist = mg.solve(b, maxit=200, tol=1e-11)
    ref, _ = O.RowsMG(p, hier=O.HIER_GEOM).fgmres(b, m=40, maxit=400, tol=1e-14)
    return ref, b, len(hist) - 1


def _check(p, xi, ref, b):
    res = np.linalg.norm(b - O.rows_apply(p, O.build_rows(p), np.ascontiguousarray(xi))) / np.linalg.norm(b)
    assert res <= 2e-11, res  # the solve's own stop at 1e-11, evaluated by the oracle's rows
    assert np.linalg.norm(xi - ref) / np.linalg.norm(ref) <= 1e-9


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("name,nu", [(n, (2, 2)) for n in CASES] + [
    ("dirichlet_ragged", (1, 1)), ("plasma_34", (1, 1)), ("plasma_33", (3, 1)), ("dirichlet_33", (1, 3)),
    ("plasma_34", (2, 0)), ("dirichlet_33", (0, 2))])
def test_relaxed_solves(handle, name, nu, prec):
    p = CASES[name]()
    ref, b, plain = _reference(p, *nu)
    dp = solver.DeviceProblem(p)
    x = torch.zeros(p.ghost_shape, dtype=torch.float64, device="cuda")
    _, info = solver.linsolve_dev(dp, x, handle=handle, tol=1e-11, precision=prec, maxit=200, nu1=nu[0], nu2=nu[1])
    assert info["status"] == 0, info
    # mixed solves go two V-cycles at a time
    assert info["vcycles"] <= plain + (2 if prec == "mixed" else 0), (info["vcycles"], plain)
    _check(p, x.cpu().numpy()[1:-1, 1:-1, 1:-1], ref, b)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_relaxed_batch(handle, prec):
    names = ["dirichlet_33", "dirichlet_ragged", "plasma_33", "plasma_34", "odd_periodic", "thin_layer", "reaction"]
    ps = [CASES[n]() for n in names]
    dps = [solver.DeviceProblem(p) for p in ps]
    xs = [torch.zeros(p.ghost_shape, dtype=torch.float64, device="cuda") for p in ps]
    infos = solver.linsolve_batched_dev(dps, xs, handle=handle, tol=1e-11, precision=prec, maxit=60)
    for p, x, info in zip(ps, xs, infos):
        assert info["status"] == 0, info
        ref, b, _ = _reference(p, 2, 2)
        _check(p, x.cpu().numpy()[1:-1, 1:-1, 1:-1], ref, b)
