"""Which top levels the cluster takes: a share of the level too large for one block
leaves it to its own launches, and a level with few planes, whose blocks are few,
sooner (cl_max_share).  Read from the profile of the level: its passes are
counted when it launches them itself.  The sizes on either side of each line are
ones that were timed both ways; the plates of the last rows ran up to 1.55 times as
long in one or two blocks as with launches of their own."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

# cells, operator, precision, whether the cluster takes the finest level
CASES = [
    ((36, 36, 36), "uniform", "fp64", True), ((33, 65, 33), "uniform", "fp64", False),
    ((42, 42, 42), "uniform", "mixed", True), ((64, 64, 16), "uniform", "mixed", False),
    ((33, 33, 33), "cell", "fp64", True), ((40, 40, 40), "cell", "fp64", False),
    ((36, 36, 36), "cell", "mixed", True), ((40, 33, 65), "cell", "mixed", False),
    ((28, 28, 28), "convection", "fp64", True), ((33, 33, 33), "convection", "fp64", False),
    ((33, 33, 33), "convection", "mixed", True), ((36, 36, 36), "convection", "mixed", False),
    ((48, 40, 6), "uniform", "fp64", True), ((150, 20, 10), "cell", "fp64", False),
    ((48, 48, 2), "uniform", "mixed", True), ((64, 64, 2), "uniform", "mixed", False),
    ((45, 50, 1), "uniform", "fp64", True), ((64, 64, 1), "uniform", "fp64", False),
    ((64, 90, 2), "uniform", "mixed", False), ((64, 64, 1), "cell", "mixed", False),
]


# the same of the second level
BELOW = [
    ((89, 89, 89), "uniform", "mixed", True), ((120, 120, 24), "uniform", "mixed", False),
    ((81, 81, 81), "cell", "mixed", True), ((116, 116, 28), "cell", "mixed", False),
    ((81, 81, 81), "convection", "mixed", True), ((116, 116, 28), "convection", "mixed", False),
    ((73, 73, 73), "uniform", "fp64", True), ((89, 89, 89), "uniform", "fp64", False),
    ((73, 73, 73), "cell", "fp64", False), ((65, 65, 65), "convection", "fp64", True),
]


@pytest.mark.parametrize("level,shape,kind,precision,cluster", [(0,) + c for c in CASES] + [(1,) + c for c in BELOW])
def test_top_level(level, shape, kind, precision, cluster):
    nx, ny, nz = shape
    rng = np.random.default_rng(6)
    g = (nz + 2, ny + 2, nx + 2)
    kw = {}
    if kind == "convection":
        kw = {"vel": rng.uniform(-1.0, 1.0, size=(3,) + g), "timederiv": True, "dt": 0.05}
    p = Problem(nx, ny, nz, (1.0, 1.0, 1.0), dcoeff=np.ones(g) if kind == "uniform" else rng.uniform(0.5, 2.0, size=g),
                source=rng.uniform(-1.0, 1.0, size=g), bc=["DIRC"] * 4 + ["ZGRD"] * 2, bcvals=[0.0] * 6, **kw)
    h = capi.Handle(0)
    h.set_profile(1 + level)
    solver.linsolve(p, handle=h, precision=precision, maxit=2, tol=1e-30,
                    krylov="fgmres" if kind == "convection" else "none")
    smoothed = h.get_profile().count[capi.PROF_SMOOTH]
    h.close()
    assert (smoothed == 0) == cluster, smoothed
