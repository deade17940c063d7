"""The Poisson solve at the sizes where the multigrid's column layout changes: columns of one lane
more or less than a warp's rows, of the most rows a lane holds in registers and beyond, levels
solved by one thread a column in shared memory, odd periodic grids smoothed by line Jacobi, long
columns that do not fit the shared-memory transposition.  The solution is checked against the
operator itself (vfs_poisson_apply): ||b - A phi|| <= 2 rtol ||b||, the solver's own acceptance of
the confirming residual, with 1e-12 of ||b|| for the rounding of the check."""
import numpy as np
import pytest

import vfs_b200 as vfs
from vfs_b200 import cases

DIMS = [(8, 8, 8), (4, 31, 6), (6, 32, 4), (12, 33, 10), (16, 64, 16), (10, 97, 8), (8, 256, 8), (8, 258, 6),
        (9, 13, 11), (7, 40, 15), (33, 16, 8), (4, 3400, 4)]


def _context(dims, seed=0, periodic_j=False):
    case = cases.channel(*dims, beta=1.0, wavy=0.05)
    if periodic_j:
        case.j_periodic, case.bctype = 1, [7] * 6
    ctx = vfs.Context(case.config())
    ctx.form_metrics(case.X, case.Y, case.Z)
    ctx.set_field(vfs.NVERT, case.nvert)
    rng = np.random.Generator(np.random.Philox(seed))
    uc = np.zeros(ctx.shape + (3,))
    uc[1:-1, 1:-1, 1:-1] = 1e-3 * rng.standard_normal((dims[2], dims[1], dims[0], 3))
    if not periodic_j:
        uc[:, -2, :, 1] = 0.0
    ctx.set_field(vfs.UCONT, uc)
    ctx.poisson_rhs()
    return ctx


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("dims", DIMS)
def test_solution_satisfies_the_operator(dims, precision):
    ctx = _context(dims)
    rtol = 1e-9
    st = ctx.poisson_solve(precision=precision, rtol=rtol, max_iter=2000, zero_guess=1)
    assert st.converged == 1
    b = ctx.get_field(vfs.B)
    r = b - ctx.poisson_apply(ctx.get_field(vfs.PHI))
    assert np.linalg.norm(r) <= (2 * rtol + 1e-12) * np.linalg.norm(b)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_periodic_columns(precision):
    """All three directions periodic: the wrap coupling of the line solves and transfers."""
    ctx = _context((16, 24, 20), periodic_j=True)
    st = ctx.poisson_solve(precision=precision, rtol=1e-9, max_iter=2000, zero_guess=1)
    assert st.converged == 1
    b = ctx.get_field(vfs.B)
    r = b - ctx.poisson_apply(ctx.get_field(vfs.PHI))
    assert np.linalg.norm(r) <= (2e-9 + 1e-12) * np.linalg.norm(b)
    ctx.close()
