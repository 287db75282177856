"""FGMRES on one handle over grids of one padded length: 8, 10 and 16 cells along x have
rows of the same pitch, but other pads.  The basis vectors that a handle keeps must
not bring the last grid's cells into the pads that the dot products run over: the
iterates equal a new handle's bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mps3d_b200 import capi, solver, workloads as W  # noqa: E402

pytestmark = pytest.mark.gpu


def _problem(nx, ny, nz, flux):
    p = W.random_operator(nx, ny, nz, bc=["DIRC", "ZGRD", "ZGRD", "ZGRD", "DIRC", "DIRC"], seed=nx, vel=True,
                          reac=False, timederiv=True)
    p.flux = flux
    return p


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("flux", [0, 1])
def test_same_padded_length(flux, precision, transpose):
    kept = capi.Handle(0)
    # the last two swap y and z
    for shape in [(16, 8, 8), (8, 8, 8), (10, 8, 8), (15, 8, 8), (8, 8, 8), (8, 16, 4), (9, 4, 16)]:
        p = _problem(*shape, flux)
        kw = dict(precision=precision, krylov="fgmres", transpose=transpose, maxit=3, tol=1e-30, restart=5)
        new = capi.Handle(0)
        want, _ = solver.linsolve(p, handle=new, **kw)
        got, _ = solver.linsolve(p, handle=kept, **kw)
        new.close()
        assert np.array_equal(got, want), (shape, np.abs(got - want).max() / np.abs(want).max())
    kept.close()
