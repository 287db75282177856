"""k_cluster's periodic z seam at the sizes whose wrapped ghost plane lies at a round
offset from the start of the neighbour block's shared memory: plane size times the
last block's planes times the word is 1024 bytes, the part of a block's shared
memory that the system keeps.  An address there must not be taken for "no
neighbour".  Against one launch per pass (MPS_SUBCYCLE=0), with test_gpu_cluster's
bounds: 1e-11 for two FP64 iterations, 1e-5 for two of a mixed solve."""
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

PER, DIR, ZG = ["PERI"] * 2, ["DIRC"] * 2, ["ZGRD"] * 2
FP64 = [(6, 6, 32), (6, 14, 16), (12, 28, 33)]
FP32 = [(6, 6, 64), (6, 14, 32), (14, 14, 8), (14, 14, 16), (24, 24, 18)]


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


@pytest.mark.parametrize("kvar", [False, True], ids=["uniform", "cell"])
@pytest.mark.parametrize("precision,shape", [("fp64", s) for s in FP64] + [("mixed", s) for s in FP32])
def test_wrapped_plane(handles, precision, shape, kvar):
    nx, ny, nz = shape
    rng = np.random.default_rng(4)
    g = (nz + 2, ny + 2, nx + 2)
    p = Problem(nx, ny, nz, (1.0, 0.8, 1.2), dcoeff=rng.uniform(0.5, 2.0, size=g) if kvar else np.full(g, 0.7),
                source=rng.uniform(-1.0, 1.0, size=g), bc=DIR + ZG + PER, bcvals=[0.3, -0.2, 0.0, 0.0, 0.0, 0.0])
    xr, _ = solver.linsolve(p, handle=handles[0], precision=precision, maxit=2, tol=1e-30)
    xc, _ = solver.linsolve(p, handle=handles[1], precision=precision, maxit=2, tol=1e-30)
    d = np.abs(xc - xr).max() / np.abs(xr).max()
    assert d <= (1e-11 if precision == "fp64" else 1e-5), d


@pytest.mark.parametrize("shape", FP64)
def test_vcycle_once(handles, shape):
    nx, ny, nz = shape
    g = (nz + 2, ny + 2, nx + 2)
    src = np.random.default_rng(5).uniform(-1.0, 1.0, size=g)
    p = Problem(nx, ny, nz, (1.0, 0.8, 1.2), dcoeff=np.ones(g), source=src, bc=DIR + ZG + PER, bcvals=[0.0] * 6)
    (xr, _), (xc, _) = [solver.vcycle_once(p, p.zeros_ghosted(), handle=h, hierarchy="geom") for h in handles]
    assert np.abs(xc - xr).max() <= 1e-11 * np.abs(xr).max()
