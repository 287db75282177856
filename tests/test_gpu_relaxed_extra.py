"""Over-relaxed passes where the diagonal extra (1/dt, a sink) weighs against the
faces: a plain pass is then nearly exact, so the relaxed schedule must give way to
it.  From an extra of a hundredth of the face sum to a thousand of them, solves take
no more V-cycles than the oracle's plain red-black Gauss-Seidel, and reach its
converged solution: the time term, a sink without one, a sink larger than the time
term in a part of the box, varying coefficients, and batches whose buffers stay while
dt changes (a replayed set-up must not keep the other schedule)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver  # noqa: E402
from mps3d_b200.problem import Problem  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

SHAPE = (33, 28, 30)
RATIOS = [0.01, 0.1, 0.16, 0.3, 1.0, 3.0, 10.0, 100.0, 1000.0]
FACES = 2.0 * sum(n * n for n in SHAPE)  # of the finest level, unit box and coefficient


@pytest.fixture(scope="module")
def handle():
    h = capi.Handle(0)
    yield h
    h.close()


def _problem(kind, ratio):
    nx, ny, nz = SHAPE
    g = (nz + 2, ny + 2, nx + 2)
    rng = np.random.default_rng(9)
    kw = {"dcoeff": np.ones(g)}
    if kind in ("dt", "cell"):
        kw.update(timederiv=True, dt=1.0 / (ratio * FACES))
    if kind == "cell":
        kw["dcoeff"] = rng.uniform(0.5, 1.0, size=g)
    if kind == "sink":
        kw["reac"] = np.full(g, -ratio * FACES) * rng.uniform(1.0, 1.2, size=g)
    if kind == "part":
        r = np.full(g, -0.1 * ratio * FACES)
        r[: g[0] // 2] *= 20.0
        kw.update(reac=r, timederiv=True, dt=1.0 / (ratio * FACES))
    return Problem(nx, ny, nz, (1.0, 1.0, 1.0), source=rng.uniform(-1.0, 1.0, size=g),
                   bc=["DIRC", "DIRC", "ZGRD", "DIRC", "ZGRD", "ZGRD"], bcvals=[0.5, 0.0, 0.0, 1.0, 0.0, 0.0], **kw)


def _plain(p, nu):
    b = O.build_rhs(p)
    _, hist = O.RowsMG(p, hier=O.HIER_GEOM, nu1=nu[0], nu2=nu[1]).solve(b, maxit=60, tol=1e-11)
    ref, _ = O.RowsMG(p, hier=O.HIER_GEOM).solve(b, maxit=60, tol=1e-15)
    return len(hist) - 1, ref


@pytest.mark.parametrize("nu", [(2, 2), (1, 1)])
@pytest.mark.parametrize("ratio", RATIOS)
@pytest.mark.parametrize("kind", ["dt", "cell", "sink", "part"])
def test_no_more_cycles_than_plain(handle, kind, ratio, nu):
    p = _problem(kind, ratio)
    plain, ref = _plain(p, nu)
    dp = solver.DeviceProblem(p)
    for precision in ("fp64", "mixed"):
        x = torch.zeros(p.ghost_shape, dtype=torch.float64, device="cuda")
        _, info = solver.linsolve_dev(dp, x, handle=handle, precision=precision, tol=1e-11, maxit=60, nu1=nu[0],
                                      nu2=nu[1])
        assert info["status"] == 0
        if precision == "fp64":
            assert info["vcycles"] <= plain, (info["vcycles"], plain)
        xi = x.cpu().numpy()[1:-1, 1:-1, 1:-1]
        assert np.linalg.norm(xi - ref) <= 1e-9 * np.linalg.norm(ref)


@pytest.mark.parametrize("kind", ["dt", "sink", "part"])
def test_batch_follows_the_extra(handle, kind):
    ratios = [0.01, 100.0, 0.1, 1000.0]
    p0 = _problem(kind, ratios[0])
    dps = [solver.DeviceProblem(_problem(kind, ratios[0])) for _ in range(2)]
    xs = [torch.zeros(p0.ghost_shape, dtype=torch.float64, device="cuda") for _ in dps]
    for ratio in [r for r in ratios for _ in range(3)]:  # the third call replays the second's set-up
        p = _problem(kind, ratio)
        plain, ref = _plain(p, (2, 2))
        for dp, x in zip(dps, xs):
            dp.prob = p
            if dp.reac is not None:
                dp.reac.copy_(torch.from_numpy(p.reac))
            x.zero_()
        infos = solver.linsolve_batched_dev(dps, xs, handle=handle, precision="fp64", tol=1e-11, maxit=30)
        for x, info in zip(xs, infos):
            assert info["status"] == 0 and info["iters"] <= -(-plain // 2), (ratio, info["iters"], plain)
            xi = x.cpu().numpy()[1:-1, 1:-1, 1:-1]
            assert np.linalg.norm(xi - ref) <= 1e-9 * np.linalg.norm(ref)
