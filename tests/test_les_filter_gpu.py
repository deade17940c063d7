"""The dynamic-Smagorinsky test filter (three one-dimensional (1 2 1) passes over tiles of 32 x 8
cells marching along k) against the C restatement, which sums the eight 2x2x2 sub-cubes as
written (rhs2.c:412-455), on grids one cell off the tile's sizes and with blocked cells.

Both sides add the same 27 non-negative-weighted products in another order: a relative 30 eps
on each filtered quantity, multiplied by the cancellation in L_ij = <U u> - <U><u> (up to 1e2
on these fields), so Cs agrees to 1e-12 of its largest value."""
import numpy as np
import pytest

from oracle import restatement
import vfs_b200 as vfs
from vfs_b200 import cases


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(31, 7, 6), (32, 8, 16), (33, 9, 17), (34, 18, 33), (4, 4, 4)])
@pytest.mark.parametrize("blocked", [False, True])
def test_filter_matches_the_restatement(dims, blocked):
    case = cases.channel(*dims, wavy=0.1)
    case.les = 2
    if blocked:
        rng = np.random.Generator(np.random.Philox(5))
        case.immersed = 1
        nv = case.nvert[1:-1, 1:-1, 1:-1]
        nv[...] = rng.choice([0, 0, 0, 0, 0, 0, 1, 3], size=nv.shape)
    m = restatement.form_metrics(case)
    u = cases.initial_ucat(case, seed=3)
    uc = cases.ucont_from_ucat(case, u, m)
    ctx = vfs.Context(case.config())
    ctx.set_metrics(m)
    ctx.set_field(vfs.NVERT, case.nvert)
    ctx.set_field(vfs.UCONT, uc)
    ctx.set_field(vfs.UCAT, u)
    ctx.set_field(vfs.UCAT_O, u)
    ctx.set_scalar(vfs.S_TI, 5)
    ctx.contra2cart()
    st = restatement.State(case, m, uc, u)
    restatement.contra2cart(st)
    np.testing.assert_array_equal(ctx.get_field(vfs.UCAT), st.ucat)
    ctx.smagorinsky_constant()
    ctx.eddy_viscosity()
    cs = restatement.les(st)
    got = ctx.get_field(vfs.CS)
    assert cs.max() > 0
    assert np.abs(got - cs).max() <= 1e-12 * cs.max()
    nut = ctx.get_field(vfs.NU_T)
    assert np.abs(nut - st.nut).max() <= 1e-12 * np.abs(st.nut).max()
    ctx.close()
