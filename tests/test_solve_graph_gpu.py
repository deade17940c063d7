"""A Poisson solve outside a step is launched kernel by kernel the first time and replayed as a
graph from the second on: the same solution bit for bit, also after the operator has been
rebuilt for other blocked cells (the graph is kept, its operands change) and with more kinds of
solves in turn than graphs are kept."""
import numpy as np
import pytest

import vfs_b200 as vfs
from vfs_b200 import cases


def _context(case, seed):
    ctx = vfs.Context(case.config())
    ctx.form_metrics(case.X, case.Y, case.Z)
    ctx.set_field(vfs.NVERT, case.nvert)
    _flow(ctx, case, seed)
    return ctx


def _flow(ctx, case, seed):
    rng = np.random.Generator(np.random.Philox(seed))
    uc = 1e-3 * rng.standard_normal(ctx.shape + (3,))
    uc[:, -2, :, 1] = 0.0
    ctx.set_field(vfs.UCONT, uc)
    ctx.volume_flux()
    ctx.poisson_rhs()


def _solve(ctx, **kw):
    st = ctx.poisson_solve(rtol=1e-9, max_iter=500, zero_guess=1, **kw)
    assert st.converged == 1
    return ctx.get_field(vfs.PHI), st.iterations


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_repeated_solves_and_a_rebuilt_operator(precision):
    case = cases.channel(20, 18, 24, wavy=0.1)
    ctx = _context(case, 1)
    first = _solve(ctx, precision=precision)
    for _ in range(3):
        again = _solve(ctx, precision=precision)
        np.testing.assert_array_equal(again[0], first[0])
        assert again[1] == first[1]
    case.nvert[8:12, 1:-1, 7:11] = 3.0
    ctx.set_field(vfs.NVERT, case.nvert)
    _flow(ctx, case, 2)
    got = _solve(ctx, precision=precision)
    fresh = _context(case, 2)
    want = _solve(fresh, precision=precision)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1] == want[1]
    fresh.close()
    ctx.close()


@pytest.mark.gpu
def test_more_kinds_of_solves_than_graphs():
    case = cases.channel(16, 12, 20)
    ctx = _context(case, 3)
    kinds = [dict(precision=p, pre_smooth=s) for p in (0, 1) for s in (1, 2, 3)]
    want = [_solve(ctx, **k)[0] for k in kinds]
    for _ in range(2):
        for k, w in zip(kinds, want):
            for _ in range(2):
                np.testing.assert_array_equal(_solve(ctx, **k)[0], w)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 2])
def test_replays_with_other_targets(precision):
    """The targets are not part of a graph: each solve stops where a fresh context's does."""
    case = cases.channel(20, 18, 24, wavy=0.1)
    ctx = _context(case, 4)
    targets = [(1e-9, 500), (1e-9, 500), (1e-4, 500), (1e-9, 3), (1e-11, 500), (1e-4, 500), (1e-9, 500)]
    for rtol, max_iter in targets:
        kw = dict(precision=precision, rtol=rtol, max_iter=max_iter, zero_guess=1, allow_unconverged=True)
        st = ctx.poisson_solve(**kw)
        fresh = _context(case, 4)
        want = fresh.poisson_solve(**kw)
        assert (st.iterations, st.converged) == (want.iterations, want.converged)
        assert st.converged == (max_iter > 3)
        np.testing.assert_array_equal(ctx.get_field(vfs.PHI), fresh.get_field(vfs.PHI))
        fresh.close()
    ctx.close()
