"""The V-cycle's small levels in one thread-block cluster (k_cluster) against one
launch per pass (a handle made with MPS_SUBCYCLE=0): both hierarchies, uniform
and cell coefficients, convection and Scharfetter-Gummel rows, transposed rows,
periodic z, merged and odd sizes, few planes, levels that one block holds, and
sweeps missing on either side.

Both forms run the same passes on the same operators in another order of
summation.  Two iterations on these small grids amplify FP64 rounding (1e-16)
by at most the condition of the coarsest solve (below 1e4): 1e-11 relative to
the largest value; the FP32 V-cycles of a mixed solve 1e-5, as the FP32 unit
6e-8 times the same growth of a cycle's few hundred operations."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver, workloads as W  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

PER, DIR, ZG = ["PERI"] * 2, ["DIRC"] * 2, ["ZGRD"] * 2


@pytest.fixture(scope="module")
def handles():
    old = os.environ.get("MPS_SUBCYCLE")
    os.environ["MPS_SUBCYCLE"] = "0"
    try:
        per_pass = capi.Handle(0)
    finally:
        if old is None:
            del os.environ["MPS_SUBCYCLE"]
        else:
            os.environ["MPS_SUBCYCLE"] = old
    cluster = capi.Handle(0)
    yield per_pass, cluster
    per_pass.close()
    cluster.close()


def _diffusion(nx, ny, nz, bc, seed=5, kvar=True, reac=False):
    rng = np.random.default_rng(seed)
    g = (nz + 2, ny + 2, nx + 2)
    shapes = [(nz, ny), (nz, ny), (nz, nx), (nz, nx), (ny, nx), (ny, nx)]
    kw = {"reac": -rng.uniform(0.5, 3.0, size=g), "timederiv": True, "dt": 0.05} if reac else {}
    return Problem(nx, ny, nz, (1.0, 0.8, 1.2), dcoeff=rng.uniform(0.5, 2.0, size=g) if kvar else np.full(g, 0.7),
                   source=rng.uniform(-1.0, 1.0, size=g), bc=bc, bcvals=[rng.uniform(-1, 1, size=s) for s in shapes],
                   **kw)


GEOM = {
    "uniform-33": lambda: _diffusion(33, 33, 33, DIR * 3, kvar=False),
    "uniform-ragged": lambda: _diffusion(41, 29, 23, DIR + ZG + ["ZGRD", "DIRC"], kvar=False),
    "uniform-periodic-z": lambda: _diffusion(24, 20, 48, ZG + DIR + PER, kvar=False),
    "cell-33": lambda: _diffusion(33, 31, 35, DIR * 3),
    "cell-all-periodic-xz": lambda: _diffusion(32, 27, 64, PER + DIR + PER),
    "few-planes": lambda: _diffusion(48, 40, 6, DIR + ZG + DIR),
    "many-planes": lambda: _diffusion(9, 10, 120, ZG + DIR + DIR),
    "one-block": lambda: _diffusion(11, 9, 10, DIR + ZG + DIR),
    "reaction": lambda: _diffusion(30, 26, 21, ZG * 3, reac=True),
}


def _pair(handles, p, **kw):
    xr, ir = solver.linsolve(p, handle=handles[0], tol=1e-30, **kw)
    xc, ic = solver.linsolve(p, handle=handles[1], tol=1e-30, **kw)
    assert ic["launches"] < ir["launches"], (ic["launches"], ir["launches"])
    return np.abs(xc - xr).max() / np.abs(xr).max()


@pytest.mark.parametrize("name,nu", [(n, (2, 2)) for n in GEOM] + [
    ("uniform-33", (0, 2)), ("cell-33", (2, 0)), ("uniform-periodic-z", (2, 0)), ("cell-all-periodic-xz", (1, 3))])
def test_geometric(handles, name, nu):
    p = GEOM[name]()
    for precision, bound in (("fp64", 1e-11), ("mixed", 1e-5)):
        d = _pair(handles, p, precision=precision, maxit=2, nu1=nu[0], nu2=nu[1])
        assert d <= bound, (precision, d)


@pytest.mark.parametrize("shape,bc,kvar", [((32, 32, 32), DIR * 3, False), ((48, 32, 16), DIR + ZG + DIR, True),
                                           ((36, 20, 28), ZG + DIR + ZG, False), ((16, 48, 64), DIR + ZG + DIR, True)])
def test_reference_hierarchy(handles, shape, bc, kvar):
    d = _pair(handles, _diffusion(*shape, bc, kvar=kvar), hierarchy="cell", precision="fp64", maxit=2)
    assert d <= 1e-11, d


@pytest.mark.parametrize("flux,transpose", [(0, False), (0, True), (1, False), (1, True)])
@pytest.mark.parametrize("shape", [(33, 29, 31), (18, 16, 40)])
def test_rows(handles, flux, transpose, shape):
    p = W.random_operator(*shape, bc=["DIRC", "ZGRD", "ZGRD", "ZGRD", "DIRC", "DIRC"], seed=3, vel=True, reac=False,
                          timederiv=True)
    p.flux = flux
    for precision, bound in (("fp64", 1e-11), ("mixed", 1e-5)):
        d = _pair(handles, p, precision=precision, krylov="fgmres", maxit=1, transpose=transpose)
        assert d <= bound, (precision, d)
