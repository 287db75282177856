"""Coefficients that are constant along most 32-cell segments of the rows: the
finest levels' passes then take one value per segment (k_kseg) and read the field
near the interfaces only.

The same problem with every cell's coefficient multiplied by 1 + 1e-13 r, r in
[-1, 1], has no two equal cells and takes the general passes.  One FP64 iteration
moves by a few times the perturbation (the operator's relative change, 1e-13,
times the factor of at most 1e2 by which a V-cycle's correction exceeds the
iterate): the iterates agree to 1e-10.  Mixed solves, whose FP32 V-cycles round
in another order, must converge alike -- the same stop within one outer iteration
-- and to a solution whose residual under the general operator (mps_apply_A_dev)
meets the stop.  Layers along each axis, a sphere, odd and merged sizes, rows
shorter than a segment's multiple, and one odd cell."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402

pytestmark = pytest.mark.gpu

PER, DIR, ZG = ["PERI"] * 2, ["DIRC"] * 2, ["ZGRD"] * 2


def _slab(shape, axis, lo, hi, v=4.0):
    k = np.ones(shape)
    idx = [slice(None)] * 3
    idx[axis] = slice(lo, hi)
    k[tuple(idx)] = v
    return k


def _sphere(shape):
    z, y, x = np.ogrid[[slice(0, n) for n in shape]]
    c = [n / 2 for n in shape]
    return np.where((z - c[0]) ** 2 + (y - c[1]) ** 2 + (x - c[2]) ** 2 < (min(shape) / 4) ** 2, 3.0, 1.0)


def _spot(shape):
    k = np.full(shape, 0.7)
    k[shape[0] // 2, 1, 31] = 1.9  # the last cell of a segment, beside a face row
    return k


# (shape z, y, x; coefficient; boundary codes; whether segments are used -- not
# with more than one change in four chunks of a row); the last two are large
# enough for the mixed solve's staged pass
CASES = [
    ("z-slab", (97, 97, 97), lambda s: _slab(s, 0, 0, 5), PER + PER + DIR, True),
    ("y-slab", (80, 90, 101), lambda s: _slab(s, 1, 40, 52), DIR + ZG + DIR, True),
    ("x-slab-thin-rows", (90, 88, 96), lambda s: _slab(s, 2, 31, 33), DIR + DIR + ZG, False),
    ("sphere", (96, 85, 83), _sphere, DIR + ZG + PER, True),
    ("spot", (81, 82, 83), _spot, ZG + DIR + ZG, True),
    ("x-interface", (94, 60, 130), lambda s: _slab(s, 2, 60, 130), DIR + DIR + ZG, True),
    ("x-slab-long-rows", (160, 150, 260), lambda s: _slab(s, 2, 60, 64), DIR + DIR + ZG, True),
    ("sphere-large", (190, 201, 193), _sphere, PER + DIR + DIR, True),
]


@pytest.fixture(scope="module")
def handle():
    h = capi.Handle(0)
    yield h
    h.close()


def _pair(shape, field, bc):
    nz, ny, nx = shape
    g = (nz + 2, ny + 2, nx + 2)
    rng = np.random.default_rng(11)
    src = rng.uniform(-1.0, 1.0, g)
    k = np.ones(g)
    k[1:-1, 1:-1, 1:-1] = field(shape)
    return [solver.DeviceProblem(Problem(nx, ny, nz, (1.0, 1.1, 0.9), dcoeff=kk, source=src, bc=bc, bcvals=[0.0] * 6))
            for kk in (k, k * (1.0 + 1e-13 * rng.uniform(-1.0, 1.0, g)))]


def _solve(dp, handle, **kw):
    x = torch.zeros(dp.prob.ghost_shape, dtype=torch.float64, device="cuda")
    return solver.linsolve_dev(dp, x, handle=handle, **kw)


@pytest.mark.parametrize("name,shape,field,bc,used", CASES, ids=[c[0] for c in CASES])
def test_fp64_iterate_matches_general_passes(handle, name, shape, field, bc, used):
    (a, ia), (b, ib) = [_solve(dp, handle, precision="fp64", tol=1e-30, maxit=1) for dp in _pair(shape, field, bc)]
    assert (ia["launches"] > ib["launches"]) == used  # the segments' own launch
    d = float((a - b).abs().max() / b.abs().max())
    assert d <= 1e-10, d


@pytest.mark.parametrize("name,shape,field,bc,used", CASES, ids=[c[0] for c in CASES])
def test_mixed_solve_converges_alike(handle, name, shape, field, bc, used):
    dps = _pair(shape, field, bc)
    (a, ia), (_, ib) = [_solve(dp, handle, precision="mixed", tol=1e-10, maxit=40) for dp in dps]
    assert ia["status"] == ib["status"] == 0
    assert abs(ia["iters"] - ib["iters"]) <= 1, (ia["iters"], ib["iters"])
    b = solver.find_bvec_dev(dps[0], handle=handle)
    r = b - solver.apply_A_dev(dps[0], a, handle=handle)
    # the solve's own residual in another order of summation: rounding of A x against b
    assert float(r.norm() / b.norm()) <= 1.1e-10
