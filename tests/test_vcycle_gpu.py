"""One multigrid V-cycle against its NumPy restatement (oracle/vcycle.py), at the sizes where the
column layout changes.  A solve of one iteration from a zero guess leaves Phi = alpha z - mean with
z = M^-1 b and alpha = <A z, b> / <A z, A z>, so the field shows every row, wrap coupling, colour and
transfer of the cycle; a check of the converged solution does not, since the outer iteration makes
up for a weaker preconditioner.

The grids have cubic cells, so the columns' line systems have a condition number of at most
`line_condition` (about 3; larger beside blocked cells).  A V-cycle is a chain of at most 80 colour
passes, each with a rounding error of a few eps times that number, and does not amplify earlier
errors: 640 eps x condition bounds the difference (2e-13 FP64, 1e-4 FP32).  A row or colour left
out changes z by more than 1e-2."""
import numpy as np
import pytest

from oracle import restatement
from oracle.vcycle import VCycle
import vfs_b200 as vfs
from vfs_b200 import cases


def _case(dims, periodic=(1, 0, 1)):
    nx, ny, nz = dims
    case = cases.channel(nx, ny, nz, beta=0.3, Lx=nx / 8, Ly=ny / 8, Lz=nz / 8, wavy=0.02)
    case.i_periodic, case.j_periodic, case.k_periodic = periodic
    case.bctype = [7 if periodic[q // 2] else 1 for q in range(6)]
    return case


def _check(case, precision, **kw):
    periodic = (case.i_periodic, case.j_periodic, case.k_periodic)
    m = restatement.form_metrics(case)
    rng = np.random.Generator(np.random.Philox(11))
    uc = np.zeros(case.da_shape + (3,))
    uc[1:-1, 1:-1, 1:-1] = 1e-3 * rng.standard_normal(uc[1:-1, 1:-1, 1:-1].shape)
    for c, ax in enumerate((2, 1, 0)):
        if not periodic[c]:
            np.moveaxis(uc[..., c], ax, 0)[-2] = 0.0
    coef = restatement.poisson_lhs(restatement.State(case, m, uc, np.zeros_like(uc)))
    ctx = vfs.Context(case.config())
    ctx.set_metrics(m)
    ctx.set_field(vfs.NVERT, case.nvert)
    ctx.set_field(vfs.UCONT, uc)
    ctx.poisson_rhs()
    b = ctx.get_field(vfs.B)
    ctx.poisson_solve(precision=precision, rtol=1e-30, max_iter=1, zero_guess=1, allow_unconverged=True, **kw)
    got = ctx.get_field(vfs.PHI)[1:-1, 1:-1, 1:-1]
    V = VCycle(coef, periodic, kw.get("pre_smooth", 3), kw.get("post_smooth", 3), kw.get("coarse_iters", 4),
               kw.get("levels", 0))
    z = np.zeros(case.da_shape)
    z[1:-1, 1:-1, 1:-1] = V.vcycle(b[1:-1, 1:-1, 1:-1])
    az = ctx.poisson_apply(z)
    ctx.close()
    want = (np.vdot(az, b) / np.vdot(az, az) * z)[1:-1, 1:-1, 1:-1]
    fluid = case.nvert[1:-1, 1:-1, 1:-1] == 0
    want = np.where(fluid, want - want[fluid].mean(), 0.0)
    eps = 2.0 ** -53 if precision == 1 else 2.0 ** -24
    assert np.isfinite(V.line_condition())
    assert np.abs(got - want).max() <= 640 * eps * V.line_condition() * np.abs(want).max()


# the whole cycle in one block; a lane more or less than a warp's rows; two to eight rows a lane and
# beyond; one thread a column and line Jacobi (odd periodic), staged and too long for shared
# memory in FP64 or both; fine levels on either side of 64^3 cells
DIMS = [(8, 8, 8), (4, 31, 6), (6, 32, 4), (12, 33, 10), (16, 64, 16), (10, 97, 8), (8, 256, 8), (8, 258, 6),
        (4, 3400, 4), (9, 13, 11), (7, 40, 15), (33, 16, 8), (5, 420, 4), (5, 900, 4), (64, 64, 64), (80, 64, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("dims", DIMS)
def test_vcycle(dims, precision):
    _check(_case(dims), precision)


@pytest.mark.gpu
def test_vcycle_of_columns_too_long_for_the_set_up_in_shared_memory():
    _check(_case((4, 12900, 4)), 1)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims,periodic", [((16, 24, 20), (1, 1, 1)), ((32, 264, 32), (1, 1, 1)), ((6, 300, 8), (0, 1, 0)),
                                           ((9, 13, 11), (0, 0, 0)), ((24, 40, 33), (1, 0, 0))])
def test_vcycle_on_other_boundaries(dims, periodic, precision):
    """Wrap couplings of periodic columns; odd cell counts that are not periodic (empty slots)."""
    _check(_case(dims, periodic), precision)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", [(16, 16, 16), (20, 40, 24), (72, 64, 64)])
def test_vcycle_with_blocked_cells(dims, precision):
    """Inactive cells and, under whole blocked columns, inactive coarse cells."""
    case = _case(dims)
    case.nvert[5:9, 1:-1, 5:9] = 3.0
    case.nvert[2:-1:7, 2:-1:5, 3:-1:6] = 3.0
    _check(case, precision)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kw", [dict(pre_smooth=1, post_smooth=2, coarse_iters=1), dict(levels=1, coarse_iters=3),
                                dict(levels=2, pre_smooth=2, post_smooth=1)])
def test_vcycle_options(kw, precision):
    _check(_case((24, 48, 32)), precision, **kw)
