"""The solver's work as its users' programs give it: the cases that are timed.

Each case is one call (or one short chain of calls) through the public entry
points on a seeded problem of the kinds that the configurations, the reference
decks and the tests of this repository use:

  poisson   constant-coefficient Poisson, Dirichlet faces (Laplace_test-style operator)
  laplace   the Laplace_test deck's boundary codes with the reference's CELL hierarchy
  gpde      one implicit step of the gpde_test deck: convection, reaction, time term
  plasma    plasma Poisson: dielectric slab, electrodes on z, periodic x/y
  electron  implicit Scharfetter-Gummel electron step, FGMRES
  batch     independent Poisson problems of uneven sizes in one batched call
  step      potential + electron part of one plasma time step
  adjoint   electron-flux loss and its gradients (torch.autograd over the solves)
  host      a plasma Poisson solve called on host arrays, as a Fortran program calls it

``exact`` solves the same systems in 64 bits without this package: the Poisson
operators are diagonalised along two axes and solved line by line along the
third; the electron systems (1/dt far above every other term) by Jacobi
iteration to rounding.
"""
import ctypes as C
import math

import numpy as np
import torch

from mps3d_b200 import adjoint, capi, solver, step, workloads
from mps3d_b200.problem import Problem

ECHARGE = 1.602176634e-19
EPS0 = 8.8541878128e-12
LENGTH = 0.01    # m: edge of the discharge box
VOLTS = 1000.0   # front electrode
# Relative residual of every solve: the parity tests' setting.  The solution is
# then determined to about 1e-10, below the last digit that a user of 1e-9 reads.
TOL = 1e-11
PERIODIC_XY = ["PERI", "PERI", "PERI", "PERI"]


def listed():
    return [
        # the smallest grid of the batch configuration, solved alone: launch latency
        {"name": "poisson_33", "kind": "poisson", "nx": 33, "ny": 33, "nz": 33, "precision": "fp64"},
        # the 65^3 configuration
        {"name": "poisson_65_mixed", "kind": "poisson", "nx": 65, "ny": 65, "nz": 65, "precision": "mixed"},
        # a box that no level divides evenly: a user's own mesh
        {"name": "poisson_ragged", "kind": "poisson", "nx": 100, "ny": 83, "nz": 61, "precision": "fp64"},
        # the reference's Laplace deck with its own hierarchy
        {"name": "laplace_128_cell", "kind": "laplace", "nx": 128, "ny": 128, "nz": 128, "precision": "fp64"},
        # the reference's generic convection-diffusion-reaction deck, one step
        {"name": "gpde_80x48x32", "kind": "gpde", "nx": 80, "ny": 48, "nz": 32, "precision": "fp64", "dt": 0.1},
        # the headline configuration in both precisions
        {"name": "plasma_257_mixed", "kind": "plasma", "nx": 257, "ny": 257, "nz": 257, "eps": 4.0,
         "precision": "mixed"},
        {"name": "plasma_257_fp64", "kind": "plasma", "nx": 257, "ny": 257, "nz": 257, "eps": 4.0,
         "precision": "fp64"},
        # the electron step configuration
        {"name": "electron_129_mixed", "kind": "electron", "nx": 129, "ny": 129, "nz": 129, "precision": "mixed",
         "dt": 1e-11},
        # the batch configuration: 64 problems of 33^3 ... 129^3
        {"name": "batch_64_mixed", "kind": "batch", "count": 64, "pick": 4, "precision": "mixed"},
        # one time step of the plasma model
        {"name": "step_129", "kind": "step", "nx": 129, "ny": 129, "nz": 129, "eps": 4.0, "dt": 1e-11},
        # one gradient of an electrode / mobility optimisation
        {"name": "adjoint_65", "kind": "adjoint", "nx": 65, "eps": 4.0, "dt": 1e-11, "steps": 5},
        # the drop-in call of a Fortran host, arrays in pageable host memory
        {"name": "host_129_mixed", "kind": "host", "nx": 129, "ny": 129, "nz": 129, "eps": 4.0,
         "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "plasma", "plasma", "laplace", "gpde", "electron", "batch", "step",
                       "adjoint", "host"])
    c = {"kind": kind}
    if kind == "batch":
        c.update(count=_log_int(rng, 2, 64), pick=rng.randrange(1000), precision=rng.choice(["mixed", "fp64"]))
        return c
    if kind == "adjoint":
        c.update(nx=_log_int(rng, 17, 97), eps=round(rng.uniform(2.0, 10.0), 2), dt=rng.choice([1e-12, 1e-11]),
                 steps=rng.randint(2, 5))
        return c
    if kind in ("laplace", "gpde"):
        # the reference halves its sizes: multiples of 16
        c.update(nx=16 * rng.randint(2, 10), ny=16 * rng.randint(2, 10), nz=16 * rng.randint(2, 10),
                 precision=rng.choice(["mixed", "fp64"]) if kind == "laplace" else "fp64")
        if kind == "gpde":
            c["dt"] = rng.choice([0.1, 0.02])
        return c
    top = {"poisson": 257, "plasma": 257, "electron": 161, "step": 145, "host": 161}[kind]
    n = _log_int(rng, 17, top)
    cube = rng.random() < 0.4
    c.update(nx=n, ny=n if cube else max(17, int(n * rng.uniform(0.6, 1.0))),
             nz=n if cube else max(17, int(n * rng.uniform(0.6, 1.0))))
    if kind in ("plasma", "step", "host"):
        c["eps"] = round(rng.uniform(2.0, 10.0), 2)
    if kind in ("electron", "step"):
        c["dt"] = rng.choice([1e-12, 1e-11])
    if kind != "step":
        c["precision"] = rng.choice(["mixed", "fp64"])
    return c


# ---- seeded fields --------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Fields:
    """Random fields of one seed, on the GPU, in the order they are asked for."""

    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, dtype=torch.float64, device=self.dev)

    def density(self, *shape):
        """lognormal(ln 1e16, 1) particles per m^3."""
        return torch.exp(math.log(1e16)
                         + torch.randn(*shape, generator=self.g, dtype=torch.float64, device=self.dev))


def _ghosted(a):
    return torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))


def _host(a):
    return a.cpu().numpy()


def _slab(case):
    """Cells of the dielectric slab: 10 of 257 along z."""
    return max(1, int(round(10 * case["nz"] / 257)))


def _eps_line(case):
    k = torch.ones(case["nz"], dtype=torch.float64, device=_device())
    k[:_slab(case)] = case["eps"]
    return k


def _eps(case):
    return _eps_line(case)[:, None, None].expand(case["nz"], case["ny"], case["nx"]).contiguous()


def _box(case):
    return (LENGTH,) * 3


def _shape(case):
    return (case["nz"], case["ny"], case["nx"])


def _problem(case, seed):
    """(Problem, exact-solver inputs) of the single-solve kinds."""
    f = _Fields(seed)
    s = _shape(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case["kind"]
    if kind == "poisson":
        return Problem(nx, ny, nz, (1.0, 1.0, 1.0), dcoeff=_host(_ghosted(torch.ones(s, dtype=torch.float64))),
                       source=_host(_ghosted(f.uniform(-1.0, 1.0, *s))), bc=["DIRC"] * 6, bcvals=[0.0] * 6)
    if kind == "laplace":
        return Problem(nx, ny, nz, (1.0, 1.0, 1.0), dcoeff=_host(_ghosted(torch.ones(s, dtype=torch.float64))),
                       source=_host(_ghosted(f.uniform(-1.0, 1.0, *s))),
                       bc=["DIRC", "DIRC"] + ["ZGRD"] * 4, bcvals=[0.0, 1.0, 0, 0, 0, 0])
    if kind == "gpde":
        return workloads.gpde_step(nx, ny, nz, phi=_host(_ghosted(f.uniform(-0.2, 0.0, *s))), dt=case["dt"])
    if kind in ("plasma", "host"):
        rho = ECHARGE / EPS0 * (f.density(*s) - f.density(*s))
        return Problem(nx, ny, nz, _box(case), dcoeff=_host(_ghosted(_eps(case))), source=_host(_ghosted(rho)),
                       bc=PERIODIC_XY + ["DIRC", "DIRC"], bcvals=[None] * 4 + [0.0, VOLTS])
    raise KeyError(kind)


def _electron_fields(case, seed):
    """(v, D, n_old / dt) of the electron step: ramp potential with a seeded ripple."""
    f = _Fields(seed)
    s = _shape(case)
    h = [LENGTH / n for n in (case["nx"], case["ny"], case["nz"])]
    z, y, x = [(torch.arange(n, dtype=torch.float64, device=f.dev) + 0.5) / n for n in s]
    amp = f.uniform(20.0, 60.0, 3)
    ph = f.uniform(0.0, 2.0 * math.pi, 3)
    ripple = (amp[0] * torch.sin(2 * math.pi * x + ph[0])[None, None, :]
              + amp[1] * torch.sin(4 * math.pi * y + ph[1])[None, :, None]
              + amp[2] * torch.sin(2 * math.pi * (x[None, :] + y[:, None]) + ph[2])[None])
    phi = VOLTS * z[:, None, None] + ripple * torch.sin(math.pi * z)[:, None, None]
    mu = 0.03 * (1.0 + f.uniform(0.0, 0.5, *s))
    te = f.uniform(1.0, 4.0, *s)
    v = mu * _gradient(phi, h, VOLTS)
    return v, mu * te, f.density(*s) / case["dt"]


def _gradient(phi, h, volts):
    """Central differences; periodic x/y, Dirichlet 0 / volts on z."""
    gx = (torch.roll(phi, -1, 2) - torch.roll(phi, 1, 2)) / (2 * h[0])
    gy = (torch.roll(phi, -1, 1) - torch.roll(phi, 1, 1)) / (2 * h[1])
    p = torch.cat([-phi[:1], phi, 2.0 * volts - phi[-1:]], dim=0)
    return torch.stack([gx, gy, (p[2:] - p[:-2]) / (2 * h[2])])


def _electron_problem(case, seed):
    v, d, b = _electron_fields(case, seed)
    return Problem(case["nx"], case["ny"], case["nz"], _box(case), dcoeff=_host(_ghosted(d)),
                   source=_host(_ghosted(b)), vel=_host(torch.stack([_ghosted(c) for c in v])),
                   bc=PERIODIC_XY + ["ZGRD", "ZGRD"], bcvals=[None] * 6, timederiv=True, dt=case["dt"], flux=1)


def _step_case(case, seed):
    f = _Fields(seed)
    s = _shape(case)
    g = lambda a: _host(_ghosted(a))  # noqa: E731
    return {"shape": (case["nx"], case["ny"], case["nz"]), "llen": _box(case), "eps": g(_eps(case)),
            "phi_bc": PERIODIC_XY + ["DIRC", "DIRC"], "phi_bcvals": [None] * 4 + [
                np.zeros((case["ny"], case["nx"])), np.full((case["ny"], case["nx"]), VOLTS)],
            "n_ion": g(f.density(*s))[None], "ion_charge": [1.0], "rho_scale": ECHARGE / EPS0,
            "ne_bc": PERIODIC_XY + ["ZGRD", "ZGRD"], "ne_bcvals": [None] * 6,
            "mu_e": g(-0.03 * (1.0 + f.uniform(0.0, 0.5, *s))), "te": g(f.uniform(1.0, 4.0, *s)), "d_e": None,
            "prod_e": None, "dt": case["dt"], "nemin": 1e7, "efield_scale": 1.0, "limiter": False,
            "scaling": (1.0, 1.0, 1.0), "n_e0": g(f.density(*s))}


def _adjoint_case(case, seed):
    f = _Fields(seed)
    n = case["nx"]
    c = dict(case, ny=n, nz=n)
    s = (n, n, n)
    rho = ECHARGE / EPS0 * (f.density(*s) - f.density(*s))
    return {"n": n, "length": LENGTH, "dt": case["dt"], "steps": case["steps"], "v_front": VOLTS,
            "eps": _host(_ghosted(_eps(c))), "rho": _host(_ghosted(rho)),
            "mu": (0.03 * (1.0 + f.uniform(0.0, 0.5, *s))).float(), "te": _host(f.uniform(1.0, 4.0, *s)),
            "n_old": _host(f.density(*s))}


def _batch(case, seed):
    ns = workloads.batch_sizes(case["count"], workloads.BATCH_SIZES, case["pick"])
    return [_problem({"kind": "poisson", "nx": n, "ny": n, "nz": n}, seed * 1009 + q) for q, n in enumerate(ns)]


# ---- the calls -------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ps = _batch(case, seed)
        return {"case": case, "dps": [solver.DeviceProblem(p) for p in ps],
                "x": [torch.zeros(p.ghost_shape, dtype=torch.float64, device="cuda") for p in ps]}
    if kind == "step":
        sc = _step_case(case, seed)
        n0 = torch.from_numpy(sc["n_e0"]).cuda()
        model = step.PlasmaStep(sc, phi_opts={"precision": "mixed", "tol": TOL, "maxit": 60},
                                e_opts={"precision": "mixed", "krylov": "fgmres", "flux": 1, "tol": TOL, "maxit": 60})
        return {"case": case, "step": model, "n0": n0, "ne": torch.zeros_like(n0), "phi": torch.zeros_like(n0)}
    if kind == "adjoint":
        ac = _adjoint_case(case, seed)
        return {"case": case, "model": adjoint.ElectronFluxAdjoint(ac), "mu": ac["mu"]}
    p = _electron_problem(case, seed) if kind == "electron" else _problem(case, seed)
    if kind == "host":
        return {"case": case, "p": p, "handle": solver.default_handle(), "x": p.zeros_ghosted()}
    return {"case": case, "dp": solver.DeviceProblem(p),
            "x": torch.zeros(p.ghost_shape, dtype=torch.float64, device="cuda")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        for x in state["x"]:
            x.zero_()
        solver.linsolve_batched_dev(state["dps"], state["x"], precision=case["precision"], tol=TOL, maxit=60)
        return state["x"]
    if kind == "step":
        state["ne"].copy_(state["n0"])
        state["phi"].zero_()
        state["step"].step(state["phi"], state["ne"])
        return {"phi": state["phi"], "ne": state["ne"]}
    if kind == "adjoint":
        loss, d_volts, d_mu = state["model"].gradient(VOLTS, state["mu"])
        return {"loss": loss, "d_volts": d_volts, "d_mu": d_mu}
    if kind == "host":
        return _host_solve(state)
    kw = {"tol": TOL, "maxit": 60, "precision": case["precision"]}
    if kind in ("laplace", "gpde"):
        kw["hierarchy"] = "cell"
    if kind == "electron":
        kw["krylov"] = "fgmres"
    x, _ = solver.linsolve_dev(state["dp"], state["x"].zero_(), **kw)
    return x


def _host_solve(state):
    """mps_linsolve as a host program calls it: NULL for the fields it does not have."""
    p, x = state["p"], state["x"]
    x[...] = 0.0
    ptr = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    g = capi.Grid(p.lx, p.ly, p.lz, *p.llen)
    o = solver.make_opts(tol=TOL, maxit=60, precision=state["case"]["precision"])
    info = capi.Info()
    st = capi.load().mps_linsolve(state["handle"].h, C.byref(g), 0, 1.0, None, ptr(p.dcoeff), None, ptr(p.source),
                                  (C.c_int * 6)(*p.bc), (C.c_void_p * 6)(*[ptr(v) for v in p.bcvals]), None, ptr(x),
                                  C.byref(o), C.byref(info))
    if st != capi.MPS_OK:
        raise capi.SolverError(st, state["handle"].last_error())
    return x


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    """Each input field read once, each output written once (8-byte words); the
    arithmetic of eleven V(2,2) cycles (1e-11 at no better than a factor of ten a
    cycle: four sweeps and a residual of 14 operations a cell, all levels)."""
    kind = case["kind"]
    cycles = 11.0 * (8.0 / 7.0) * 5 * 14
    if kind == "batch":
        n = sum(m ** 3 for m in workloads.batch_sizes(case["count"], workloads.BATCH_SIZES, case["pick"]))
        return {"bytes": 8.0 * 3 * n, "flops": cycles * n}
    if kind == "adjoint":
        n = case["nx"] ** 3
        # eps, b0, b1, Te, n_old, mobility in, its gradient out; the states kept between the passes
        return {"bytes": 8.0 * (5 + 2 * case["steps"]) * n + 8.0 * n,
                "flops": (2 * cycles + 2 * case["steps"] * cycles / 10) * n}
    n = case["nx"] * case["ny"] * case["nz"]
    words = {"poisson": 3, "laplace": 3, "plasma": 3, "host": 3, "gpde": 7, "electron": 6, "step": 14}[kind]
    scale = {"electron": 0.2, "step": 1.2}.get(kind, 1.0)
    return {"bytes": 8.0 * words * n, "flops": scale * cycles * n}


# ---- the same in 64 bits, without the package --------------------------------

def _axis_matrix(n, h, lo, hi):
    """-d2/dx2 of n cells of width h: 'PERI', 'DIRC' (face value) or 'ZGRD' ends."""
    a = np.zeros((n, n))
    for i in range(n):
        for j, end in ((i - 1, lo), (i + 1, hi)):
            if 0 <= j < n:
                a[i, i] += 1 / h ** 2
                a[i, j] -= 1 / h ** 2
            elif end == "PERI":
                a[i, i] += 1 / h ** 2
                a[i, j % n] -= 1 / h ** 2
            elif end == "DIRC":
                a[i, i] += 2 / h ** 2
    return a


def _line_solve(b, ka, ma, mb, lower, diag, upper):
    """u of (k(l) (Ma + Mb) + T) u = b, axes (l, a, b): Ma, Mb symmetric, T
    tridiagonal along l (lower, diag, upper), k a line of coefficients."""
    dev = b.device
    wa, qa = [torch.from_numpy(v).to(dev) for v in np.linalg.eigh(ma)]
    wb, qb = [torch.from_numpy(v).to(dev) for v in np.linalg.eigh(mb)]
    r = torch.matmul(torch.matmul(qa.T, b), qb)
    lam = wa[:, None] + wb[None, :]
    n = b.shape[0]
    lower, diag, upper, ka = [np.asarray(v, dtype=np.float64) for v in (lower, diag, upper, ka)]
    cp = [None] * n
    for i in range(n):
        d = diag[i] + ka[i] * lam
        if i:
            d = d - lower[i] * cp[i - 1]
            r[i] -= lower[i] * r[i - 1]
        cp[i] = upper[i] / d
        r[i] /= d
    for i in range(n - 2, -1, -1):
        r[i] -= cp[i] * r[i + 1]
    return torch.matmul(torch.matmul(qa, r), qb.T)


def _diffusion(k, h, lo, hi):
    """Tridiagonal -d(k d)/dx with arithmetic face means and 'DIRC' or 'ZGRD' ends."""
    n = len(k)
    lower, diag, upper = np.zeros(n), np.zeros(n), np.zeros(n)
    for i in range(n):
        for j, end, off in ((i - 1, lo, lower), (i + 1, hi, upper)):
            if 0 <= j < n:
                w = 0.5 * (k[i] + k[j]) / h ** 2
                diag[i] += w
                off[i] = -w
            elif end == "DIRC":
                diag[i] += 2 * k[i] / h ** 2
    return lower, diag, upper


def _plasma_exact(case, rhs):
    """Potential of a right-hand side that holds its boundary terms already."""
    h = [LENGTH / n for n in (case["nx"], case["ny"], case["nz"])]
    k = _host(_eps_line(case))
    return _line_solve(rhs, k, _axis_matrix(case["ny"], h[1], "PERI", "PERI"),
                       _axis_matrix(case["nx"], h[0], "PERI", "PERI"), *_diffusion(k, h[2], "DIRC", "DIRC"))


def _front(case, volts):
    """Boundary term of the front electrode in the right-hand side."""
    b = torch.zeros(_shape(case), dtype=torch.float64, device=_device())
    b[-1] = 2.0 * float(_eps_line(case)[-1]) * volts / (LENGTH / case["nz"]) ** 2
    return b


def _sg_weights(c_l, c_r, d_l, d_r, h):
    """Scharfetter-Gummel face flux w_l u_l + w_r u_r."""
    d = 2.0 * d_l * d_r / (d_l + d_r + 1e-10)
    pe = 0.5 * (c_l + c_r) * h / d
    bern = lambda x: x / torch.expm1(x)  # noqa: E731
    return d / h * bern(-pe), -d / h * bern(pe)


def _sg_rows(v, d, h, dt):
    """Diagonal and the six neighbour coefficients; periodic x/y, ZGRD z."""
    diag = torch.full_like(d, 1.0 / dt)
    co = []
    for ax, dim in ((0, 2), (1, 1)):
        wl, wr = _sg_weights(v[ax], torch.roll(v[ax], -1, dim), d, torch.roll(d, -1, dim), h[ax])
        diag = diag + wl / h[ax] - torch.roll(wr, 1, dim) / h[ax]
        co += [-torch.roll(wl, 1, dim) / h[ax], wr / h[ax]]
    wl, wr = _sg_weights(v[2][:-1], v[2][1:], d[:-1], d[1:], h[2])
    zero = torch.zeros_like(d[:1])
    # the end cells: convective outflow only
    diag = diag + torch.cat([wl, v[2][-1:]]) / h[2] - torch.cat([v[2][:1], wr]) / h[2]
    co += [-torch.cat([zero, wl]) / h[2], torch.cat([wr, zero]) / h[2]]
    return diag, co


def _sg_solve(rows, b):
    diag, co = rows
    x = b / diag
    zero = torch.zeros_like(b[:1])
    for _ in range(14):  # off-diagonal over diagonal below 0.05 at every size and dt above
        off = (co[0] * torch.roll(x, 1, 2) + co[1] * torch.roll(x, -1, 2) + co[2] * torch.roll(x, 1, 1)
               + co[3] * torch.roll(x, -1, 1) + co[4] * torch.cat([zero, x[:-1]])
               + co[5] * torch.cat([x[1:], zero]))
        x = (b - off) / diag
    return x


def _inner(p):
    return torch.from_numpy(p).to(_device())[1:-1, 1:-1, 1:-1]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ns = workloads.batch_sizes(case["count"], workloads.BATCH_SIZES, case["pick"])
        return [exact({"kind": "poisson", "nx": n, "ny": n, "nz": n}, seed * 1009 + q) for q, n in enumerate(ns)]
    if kind == "adjoint":
        return _adjoint_exact(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "electron":
        v, d, b = _electron_fields(case, seed)
        return _ghosted(_sg_solve(_sg_rows(v, d, [LENGTH / nx, LENGTH / ny, LENGTH / nz], case["dt"]), b))
    if kind == "step":
        return _step_exact(case, seed)
    p = _problem(case, seed)
    b = _inner(p.source)
    if kind in ("plasma", "host"):
        x = _ghosted(_plasma_exact(case, b + _front(case, VOLTS)))
        return _host(x) if kind == "host" else x
    if kind == "poisson":
        one = np.ones(nz)
        return _ghosted(_line_solve(b, one, _axis_matrix(ny, 1.0 / ny, "DIRC", "DIRC"),
                                    _axis_matrix(nx, 1.0 / nx, "DIRC", "DIRC"),
                                    *_diffusion(one, 1.0 / nz, "DIRC", "DIRC")))
    # laplace, gpde: lines along x
    b = b.permute(2, 0, 1).contiguous()
    h = [length / n for length, n in zip(p.llen, (nx, ny, nz))]
    k = np.full(nx, 1.0 if kind == "laplace" else 0.5)
    if kind == "laplace":
        lower, diag, upper = _diffusion(k, h[0], "DIRC", "DIRC")
        b[-1] += 2.0 / h[0] ** 2
    else:
        lower, diag, upper = _diffusion(k, h[0], "DIRC", "FLUX")
        # drift -1: the right cell of a face is upwind; the left wall lets it out
        diag += 1 / h[0] - 2.0 + 1.0 / case["dt"]
        upper[:-1] -= 1 / h[0]
        b[-1] += 0.25 / h[0]
    u = _line_solve(b, k, _axis_matrix(nz, h[2], "ZGRD", "ZGRD"), _axis_matrix(ny, h[1], "ZGRD", "ZGRD"),
                    lower, diag, upper)
    return _ghosted(u.permute(1, 2, 0).contiguous())


def _faces(u, lo, hi):
    """u with its face ghosts: periodic x/y, given planes on z."""
    g = _ghosted(u)
    g[1:-1, 1:-1, 0], g[1:-1, 1:-1, -1] = u[:, :, -1], u[:, :, 0]
    g[1:-1, 0, 1:-1], g[1:-1, -1, 1:-1] = u[:, -1, :], u[:, 0, :]
    g[0, 1:-1, 1:-1], g[-1, 1:-1, 1:-1] = lo, hi
    return g


def _step_exact(case, seed):
    sc = _step_case(case, seed)
    h = [LENGTH / n for n in (case["nx"], case["ny"], case["nz"])]
    n_old, mu, te = _inner(sc["n_e0"]), _inner(sc["mu_e"]), _inner(sc["te"])
    phi = _plasma_exact(case, sc["rho_scale"] * (_inner(sc["n_ion"][0]) - n_old) + _front(case, VOLTS))
    rows = _sg_rows(-mu * _gradient(phi, h, VOLTS), -mu * te, h, case["dt"])
    ne = torch.clamp(_sg_solve(rows, n_old / case["dt"]), min=sc["nemin"])
    return {"phi": _faces(phi, -phi[0], 2.0 * VOLTS - phi[-1]), "ne": _faces(ne, ne[0], ne[-1])}


def _adjoint_exact(case, seed):
    ac = _adjoint_case(case, seed)
    n = case["nx"]
    c = dict(case, ny=n, nz=n)
    h = LENGTH / n
    phi0 = _plasma_exact(c, _inner(ac["rho"]))
    phi1 = _plasma_exact(c, _front(c, 1.0))
    te, n_old = [torch.from_numpy(ac[q]).to(_device()) for q in ("te", "n_old")]
    volts = torch.tensor(VOLTS, dtype=torch.float64, device=te.device, requires_grad=True)
    mu = ac["mu"].clone().requires_grad_(True)
    m = mu.double()
    v = m * _gradient(phi0 + volts * phi1, [h, h, h], volts)
    rows = _sg_rows(v, m * te, [h, h, h], case["dt"])
    ne = n_old
    for _ in range(case["steps"]):
        ne = _sg_solve(rows, ne / case["dt"])
    loss = (v[2, -1] * ne[-1]).sum() * h * h
    g_volts, g_mu = torch.autograd.grad(loss, (volts, mu))
    return {"loss": float(loss.detach()), "d_volts": float(g_volts), "d_mu": g_mu}
