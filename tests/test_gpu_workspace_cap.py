"""A handle under MPS_WORKSPACE_LIMIT_BYTES does without the arrays that only buy time
-- the cluster's rows, uniform segments, averaged-face coarse coefficients, the
transposed rows' scratch -- before it refuses a grid.  The caps are what each solve
needs without them (to the next KiB), and half of that is still refused."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver, workloads as W  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu


def _slab(n):
    g = (n + 2,) * 3
    k = np.ones(g)
    k[:8] = 4.0
    return Problem(n, n, n, (1.0, 1.0, 1.0), dcoeff=k, source=np.random.default_rng(0).uniform(-1.0, 1.0, g),
                   bc=["PERI"] * 4 + ["DIRC"] * 2, bcvals=[0.0] * 6)


def _cell(n):
    g = (n + 2,) * 3
    return Problem(n, n, n, (1.0, 1.0, 1.0), dcoeff=np.random.default_rng(1).uniform(0.5, 2.0, g), source=np.ones(g),
                   bc=["DIRC"] * 6, bcvals=[0.0] * 6)


def _convection(n):
    return W.random_operator(n, n, n, bc=["DIRC", "ZGRD", "ZGRD", "ZGRD", "DIRC", "DIRC"], seed=3, vel=True,
                             reac=False, timederiv=True)


CASES = {
    "slab-81": (lambda: _slab(81), {}, 54807282),
    "cell-33": (lambda: _cell(33), {}, 4731619),
    "transposed-33": (lambda: _convection(33), {"krylov": "fgmres", "transpose": True, "restart": 5}, 10552703),
    "convection-33": (lambda: _convection(33), {"krylov": "fgmres", "restart": 5}, 10552703),
}


def _handle(monkeypatch, cap):
    monkeypatch.setenv("MPS_WORKSPACE_LIMIT_BYTES", str(cap))
    h = capi.Handle(0)
    monkeypatch.delenv("MPS_WORKSPACE_LIMIT_BYTES")
    return h


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", CASES)
def test_solves_under_the_cap(monkeypatch, name, precision):
    make, kw, cap = CASES[name]
    p = make()
    kw = dict(kw, precision=precision, tol=1e-10, maxit=60)
    free, capped = capi.Handle(0), _handle(monkeypatch, cap)
    want, _ = solver.linsolve(p, handle=free, **kw)
    for _ in range(2):  # also with the workspace in place
        got, info = solver.linsolve(p, handle=capped, **kw)
        assert info["status"] == 0
        # both stop at a relative residual of 1e-10; these operators' condition is below 1e4
        assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    free.close()
    capped.close()


@pytest.mark.parametrize("name", CASES)
def test_half_of_it_is_refused(monkeypatch, name):
    make, kw, cap = CASES[name]
    h = _handle(monkeypatch, cap // 2)
    with pytest.raises(capi.SolverError) as e:
        solver.linsolve(make(), handle=h, **kw)
    assert e.value.status == capi.MPS_ERR_NOMEM
    _, info = solver.linsolve(W.poisson_dirichlet(9), handle=h)
    assert info["status"] == 0
    h.close()
