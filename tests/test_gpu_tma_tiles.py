"""The staged colour pass (k_colour_tma) at sizes that reach it: chunks of at least
eight planes, in both tile forms -- six rows with a staged coefficient, eight rows
with a uniform one or one along most rows -- against the register-fed pass of a handle
made with MPS_TMA=0.  Odd and even periodic seams, zero-gradient and Dirichlet
faces, merged sizes, rows and planes that do not divide into the tiles, rows of
several lane groups; V(2,2) cycles on both sides, so plain and over-relaxed passes.

Both forms evaluate a cell in the same order, so two iterations agree up to the
compiler's contraction choices in FP32: 1e-6 of the largest value, as in
test_gpu_tma.  That the staged kernel is what runs is read from a trace of its
launches, taken in a process of its own (this file as a program)."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from mps3d_b200 import capi, solver  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

PER, DIR, ZG = ["PERI"] * 2, ["DIRC"] * 2, ["ZGRD"] * 2


def _problem(shape, bc, kind):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx)
    g = (nz + 2, ny + 2, nx + 2)
    k = np.full(g, 0.8)
    if kind == "cell":
        k = rng.uniform(0.5, 2.0, size=g)
    elif kind == "segments":
        k[:, 1 + ny // 3:1 + ny // 3 + 9, :] = 3.0
        k[nz // 2, ny // 2, nx // 2] = 1.7
    elif kind == "x-layer":  # no row has one coefficient: the field is staged
        k[:, :, : nx // 3] = 3.0
    elif kind == "x-block":  # a fifth of the planes
        k[: nz // 5, :, : nx // 3] = 3.0
    return Problem(nx, ny, nz, (1.0, 0.8, 1.2), dcoeff=k, source=rng.uniform(-1.0, 1.0, size=g), bc=bc,
                   bcvals=[0.0, 0.4, 0.0, 0.0, -0.3, 0.0])


# (cells x, y, z; boundary codes; coefficient; rows of the tile that must run)
CASES = {
    "cell-odd-periodic": ((45, 157, 149), PER * 3, "cell", 6),
    "cell-mixed-faces": ((36, 150, 160), PER + DIR + ["ZGRD", "DIRC"], "cell", 6),
    "cell-merged": ((57, 163, 141), ["ZGRD", "DIRC"] + DIR + ZG, "cell", 6),
    "cell-long-rows": ((330, 146, 152), DIR + PER + ZG, "cell", 6),
    "uniform-odd-periodic": ((33, 205, 203), PER * 3, "uniform", 8),
    "uniform-dirichlet": ((40, 200, 212), DIR * 3, "uniform", 8),
    "uniform-ragged": ((27, 221, 191), ["DIRC", "ZGRD"] + ZG + PER, "uniform", 8),
    "segments-odd-periodic": ((45, 205, 203), PER * 3, "segments", 8),
    "segments-mixed-faces": ((70, 198, 216), ZG + DIR + PER, "segments", 8),
    "x-layer": ((128, 160, 150), PER + DIR + ZG, "x-layer", 6),
    "x-block": ((130, 203, 207), PER + PER + DIR, "x-block", 8),
    "segments-long-rows": ((301, 197, 201), DIR + ["DIRC", "ZGRD"] + DIR, "segments", 8),
}


@pytest.fixture(scope="module")
def handles():
    old = os.environ.get("MPS_TMA")
    os.environ["MPS_TMA"] = "0"
    try:
        reg = capi.Handle(0)
    finally:
        if old is None:
            del os.environ["MPS_TMA"]
        else:
            os.environ["MPS_TMA"] = old
    tma = capi.Handle(0)
    yield reg, tma
    reg.close()
    tma.close()


@pytest.fixture(scope="module")
def launched():
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.splitlines()[-1])


@pytest.mark.parametrize("name", CASES)
def test_staged_pass_runs(launched, name):
    rows = CASES[name][3]
    assert any(f"k_colour_tma<float, 4, {rows}," in k for k in launched[name]), launched[name]


@pytest.mark.parametrize("nu", [(2, 2), (1, 1), (3, 1)])
@pytest.mark.parametrize("name", CASES)
def test_staged_pass_matches_register_pass(handles, name, nu):
    shape, bc, kind, _ = CASES[name]
    dp = solver.DeviceProblem(_problem(shape, bc, kind))
    xs = []
    for h in handles:
        x = torch.zeros(dp.prob.ghost_shape, dtype=torch.float64, device="cuda")
        xs.append(solver.linsolve_dev(dp, x, handle=h, precision="mixed", maxit=2, tol=1e-30, nu1=nu[0], nu2=nu[1])[0])
    d = float((xs[1] - xs[0]).abs().max() / xs[0].abs().max())
    print(f"{name}: staged against register-fed colour pass, largest relative difference {d:.3e}")
    assert d <= 1e-6, d


def _trace():
    from torch.profiler import ProfilerActivity, profile

    out = {}
    h = capi.Handle(0)
    for name, (shape, bc, kind, _) in CASES.items():
        dp = solver.DeviceProblem(_problem(shape, bc, kind))
        x = torch.zeros(dp.prob.ghost_shape, dtype=torch.float64, device="cuda")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            solver.linsolve_dev(dp, x, handle=h, precision="mixed", maxit=1, tol=1e-30, use_graph=0)
            torch.cuda.synchronize()
        out[name] = sorted({e.name for e in prof.events() if "k_colour" in e.name})
    print(json.dumps(out))


if __name__ == "__main__":
    _trace()
