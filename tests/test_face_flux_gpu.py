"""Formfunction_2 with its face fluxes split between the interior form and the listed faces of
boundary and body points, against the C restatement, bit for bit: grids with no, one and few
interior-form points, one point off a block of 128, without bodies and with random blocked or
immersed cells, and a second nvert field on the same context (the list grows, then shrinks)."""
import numpy as np
import pytest

from oracle import restatement
import vfs_b200 as vfs
from vfs_b200 import cases


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(4, 4, 4), (5, 5, 5), (6, 5, 7), (30, 9, 11), (33, 12, 10)])
@pytest.mark.parametrize("periodic", [(1, 0, 1), (0, 0, 0)])
@pytest.mark.parametrize("immersed", [0, 1])
def test_formfunction2_matches_the_restatement(dims, periodic, immersed):
    case = cases.channel(*dims, wavy=0.1)
    case.i_periodic, case.j_periodic, case.k_periodic = periodic
    if not periodic[0]:
        case.bctype = [1] * 6
    case.immersed = immersed
    m = restatement.form_metrics(case)
    u = cases.initial_ucat(case, seed=3)
    uc = cases.ucont_from_ucat(case, u, m)
    ctx = vfs.Context(case.config())
    ctx.set_metrics(m)
    rng = np.random.Generator(np.random.Philox(7))
    for values in ([0], [0] * 30 + [1, 3], [0, 0, 1, 3], [0]):
        nv = np.zeros_like(case.nvert)
        nv[1:-1, 1:-1, 1:-1] = rng.choice(values, size=nv[1:-1, 1:-1, 1:-1].shape)
        case.nvert = nv
        ctx.set_field(vfs.NVERT, nv)
        ctx.set_field(vfs.UCONT, uc)
        ctx.set_field(vfs.UCAT, u)
        ctx.set_field(vfs.UCAT_O, u)
        ctx.contra2cart()
        st = restatement.State(case, m, uc, u)
        restatement.contra2cart(st)
        rhs0 = rng.standard_normal(u.shape)
        ctx.set_field(vfs.RHS, rhs0)
        ctx.formfunction2(1.0)
        want = restatement.formfunction2(st, 1.0, rhs=rhs0)
        np.testing.assert_array_equal(ctx.get_field(vfs.RHS), want)
    ctx.close()
