"""One handle, the same cells and boundary codes in another box: every face
coefficient scales with the cell widths, so nothing that a handle keeps between
calls (captured iterations, the cluster's tables) may carry the first box's.

The handle that solved in the first box must give what a new handle gives, bit for
bit: both run the same launches on the same data."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver, workloads as W  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

DIR, ZG, PER = ["DIRC"] * 2, ["ZGRD"] * 2, ["PERI"] * 2
BOXES = [(1.0, 1.0, 1.0), (0.01, 0.02, 0.01), (1.0, 1.0, 1.3), (1.0, 1.0, 1.0)]


def _diffusion(shape, bc, kvar, llen):
    nx, ny, nz = shape
    rng = np.random.default_rng(2)
    g = (nz + 2, ny + 2, nx + 2)
    return Problem(nx, ny, nz, llen, dcoeff=rng.uniform(0.5, 2.0, size=g) if kvar else np.ones(g),
                   source=rng.uniform(-1.0, 1.0, size=g), bc=bc, bcvals=[0.0, 1.0, 0.5, 0.0, 0.0, -1.0])


def _convection(llen):
    p = W.random_operator(24, 20, 28, bc=["DIRC", "ZGRD", "ZGRD", "ZGRD", "DIRC", "DIRC"], seed=3, vel=True,
                          reac=False, timederiv=True)
    p.llen = llen
    return p


CASES = {
    "uniform-33": (lambda b: _diffusion((33, 33, 33), DIR * 3, False, b), {}),
    "uniform-65": (lambda b: _diffusion((65, 65, 65), DIR * 3, False, b), {}),
    "cell-periodic": (lambda b: _diffusion((40, 36, 44), PER + DIR + ZG, True, b), {}),
    "reference-hierarchy": (lambda b: _diffusion((32, 48, 32), DIR + ZG + DIR, False, b), {"hierarchy": "cell"}),
    "convection": (_convection, {"krylov": "fgmres"}),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("opts", [{}, {"use_graph": 0}, {"nu1": 2, "nu2": 1}], ids=["graph", "no-graph", "odd-sweeps"])
@pytest.mark.parametrize("name", CASES)
def test_second_box_on_one_handle(name, opts, precision):
    make, kw = CASES[name]
    kw = dict(kw, precision=precision, maxit=2, tol=1e-30, **opts)
    kept = capi.Handle(0)
    for box in BOXES:
        p = make(box)
        new = capi.Handle(0)
        want, _ = solver.linsolve(p, handle=new, **kw)
        got, _ = solver.linsolve(p, handle=kept, **kw)
        new.close()
        assert np.array_equal(got, want), (box, np.abs(got - want).max() / np.abs(want).max())
    kept.close()


@pytest.mark.parametrize("name", ["uniform-33", "uniform-65", "reference-hierarchy"])
def test_vcycle_once_in_a_second_box(name):
    make, kw = CASES[name]
    kept = capi.Handle(0)
    for box in BOXES:
        p = make(box)
        new = capi.Handle(0)
        want, rw = solver.vcycle_once(p, p.zeros_ghosted(), handle=new, **kw)
        got, rg = solver.vcycle_once(p, p.zeros_ghosted(), handle=kept, **kw)
        new.close()
        assert np.array_equal(got, want) and rg == rw, (box, rg, rw)
    kept.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_in_a_second_box(precision):
    bound = 1e-11 if precision == "fp64" else 1e-5
    kept = capi.Handle(0)
    for box in BOXES:
        dps = [solver.DeviceProblem(CASES[n][0](box)) for n in ("uniform-33", "cell-periodic")]
        out = []
        for h in (capi.Handle(0), kept):
            xs = [torch.zeros(d.prob.ghost_shape, dtype=torch.float64, device="cuda") for d in dps]
            solver.linsolve_batched_dev(dps, xs, handle=h, precision=precision, maxit=2, tol=1e-30)
            out.append(xs)
        for a, b in zip(*out):  # (each handle times its own launch shapes: rounding of two V-cycles apart)
            assert float((a - b).abs().max()) <= bound * float(b.abs().max()), box
    kept.close()
