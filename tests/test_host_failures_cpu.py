"""What the host code does when a CUDA call fails, on a CUDA runtime in host memory whose calls fail
on request: the failure is reported, and a call after it neither uses what was not allocated nor
forgets to allocate it."""
import pytest

import vfs_b200 as vfs
from vfs_b200 import cases
from fake_cuda import context, fake, fake_library  # noqa: F401

ERR_CUDA = 2


@pytest.mark.parametrize("kernel", ["k_face_flux", "k_fp", "k_rhs", "k_periodic_copy"])
def test_a_failed_launch_of_formfunction2_is_reported(fake, kernel):
    ctx = context()
    ctx.formfunction2(1.0)
    fake.fake_fail_kernel(kernel.encode())
    with pytest.raises(vfs.VfsError) as e:
        ctx.formfunction2(1.0)
    assert kernel in str(e.value)
    fake.fake_fail_kernel(b"")
    ctx.formfunction2(1.0)
    ctx.close()


@pytest.mark.parametrize("kernel,which", [("k_face_flux", 0), ("k_fp", 1), ("k_rhs", 2), ("k_zcol", 4)])
def test_a_failed_launch_of_a_single_kernel_is_reported(fake, kernel, which):
    ctx = context()
    ctx.poisson_lhs()
    ctx.run_kernel(which)
    fake.fake_fail_kernel(kernel.encode())
    with pytest.raises(vfs.VfsError):
        ctx.run_kernel(which)
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_a_solve_after_a_failed_allocation_allocates_what_is_missing(fake, precision):
    """Each allocation of the first solve fails in turn; the same solve again allocates the rest."""
    ctx = context()
    ctx.poisson_rhs()
    n0 = fake.fake_mallocs()
    ctx.poisson_solve(precision=precision, allow_unconverged=True)
    need = fake.fake_mallocs() - n0
    assert need >= 2
    ctx.close()
    for nth in range(1, need + 1):
        ctx = context()
        ctx.poisson_rhs()
        fake.fake_fail_malloc(nth)
        with pytest.raises(vfs.VfsError) as e:
            ctx.poisson_solve(precision=precision, allow_unconverged=True)
        assert "allocation" in str(e.value)
        with pytest.raises(vfs.VfsError) as e:  # still no memory: nothing may be launched without its buffers
            ctx.poisson_solve(precision=precision, allow_unconverged=True)
        assert "allocation" in str(e.value)
        fake.fake_fail_malloc(0)
        n0 = fake.fake_mallocs()
        ctx.poisson_solve(precision=precision, allow_unconverged=True)
        assert fake.fake_mallocs() - n0 == need - nth + 1
        ctx.close()


def test_an_operator_after_a_failed_allocation_allocates_what_is_missing(fake):
    """Each allocation of the operator and its multigrid levels fails in turn."""
    ctx = context()
    ctx.form_bcs()  # what is allocated on the way (reduction buffer, point lists) is there
    ctx.poisson_lhs()
    ctx.close()
    ctx = context()
    ctx.form_bcs()
    n0 = fake.fake_mallocs()
    ctx.poisson_lhs()
    need = fake.fake_mallocs() - n0
    assert need > 15  # the operator's five, six or seven a level
    ctx.close()
    for nth in range(1, need + 1):
        ctx = context()
        ctx.form_bcs()
        fake.fake_fail_malloc(nth)
        for _ in range(2):
            with pytest.raises(vfs.VfsError) as e:
                ctx.poisson_lhs()
            assert "allocation" in str(e.value)
        fake.fake_fail_malloc(0)
        ctx.poisson_lhs()
        ctx.poisson_rhs()
        ctx.poisson_solve(allow_unconverged=True)
        n0 = fake.fake_mallocs()
        ctx.poisson_lhs()
        assert fake.fake_mallocs() == n0
        ctx.close()


def test_no_reduction_without_its_buffer(fake):
    """The solve asks for a larger reduction buffer; when that fails the old one is gone."""
    ctx = context()
    ctx.poisson_rhs()
    ctx.poisson_solve(allow_unconverged=True, precision=0)
    ctx.close()
    ctx = context()
    ctx.poisson_rhs()
    fake.fake_fail_malloc(3)  # after the basis and the preconditioned vectors
    with pytest.raises(vfs.VfsError) as e:
        ctx.poisson_solve(allow_unconverged=True, precision=0)
    assert "reduction buffer" in str(e.value)
    with pytest.raises(vfs.VfsError) as e:
        ctx.divergence()
    assert "reduction buffer" in str(e.value)
    assert fake.fake_launches(b"k_divergence") == 0
    fake.fake_fail_malloc(0)
    ctx.divergence()
    ctx.close()


@pytest.mark.parametrize("precision,size", [(0, 4), (1, 8), (2, 4)])
def test_the_first_solve_clears_no_more_than_the_preconditioned_vectors(fake, precision, size):
    """Their ghost points are never written; the basis is written whole before it is read."""
    ctx = context()
    ctx.poisson_rhs()
    n0 = fake.fake_cleared_bytes()
    ctx.poisson_solve(precision=precision, restart=20, allow_unconverged=True)
    n = ctx.shape[0] * ctx.shape[1] * ctx.shape[2]
    ld = (n + 31) // 32 * 32
    assert fake.fake_cleared_bytes() - n0 == 20 * ld * size + 8 * n  # and Phi, the zero guess
    ctx.close()


def test_solves_that_differ_in_their_targets_share_a_graph(fake):
    """A caller who changes the tolerance every two solves does not pay a capture for each replay."""
    ctx = context()
    ctx.poisson_rhs()
    kw = dict(zero_guess=1, allow_unconverged=True)
    for rtol in (1e-4, 1e-6, 1e-8):
        for max_iter in (50, 100):
            for _ in range(2):
                ctx.poisson_solve(rtol=rtol, max_iter=max_iter, **kw)
    assert (fake.fake_captures(), fake.fake_graph_launches()) == (1, 11)
    ctx.poisson_solve(rtol=1e-8, max_iter=100, pre_smooth=2, **kw)
    ctx.poisson_solve(rtol=1e-8, max_iter=100, pre_smooth=2, **kw)
    assert (fake.fake_captures(), fake.fake_graph_launches()) == (2, 12)
    ctx.close()


def test_precisions_in_turn_where_memory_holds_one(fake):
    """The vectors of another precision are given back when a solve's own do not fit: a context that
    alternates between the precisions needs no more memory than its largest."""
    need = {}
    for precision in (0, 1, 2):
        ctx = context()
        ctx.poisson_rhs()
        ctx.poisson_solve(precision=precision, allow_unconverged=True)
        need[precision] = fake.fake_allocated()
        ctx.close()
    ctx = context()
    ctx.poisson_rhs()
    fake.fake_limit(need[1])
    for precision in (0, 1, 2, 1, 0, 2, 0):
        ctx.poisson_solve(precision=precision, allow_unconverged=True)
        assert fake.fake_allocated() <= need[1]
    n0 = fake.fake_mallocs()
    ctx.poisson_solve(precision=0, allow_unconverged=True)  # nothing is given back while it fits
    assert fake.fake_mallocs() == n0
    ctx.close()


@pytest.mark.parametrize("nth", [2, 3, 4, 5])
def test_point_lists_after_a_search_that_failed_half_way(fake, nth):
    """The ray casting has written nvert by then: the lists of boundary and body points that
    Contra2Cart and the face fluxes run over, and the Poisson operator, are not those any more."""
    ctx = context(immersed=1)
    ctx.poisson_lhs()
    ctx.contra2cart()
    ctx.formfunction2(1.0)
    lists, operators = (fake.fake_launches(k) for k in (b"k_collect_points", b"k_poisson_coef"))
    ctx.formfunction2(1.0)
    assert fake.fake_launches(b"k_collect_points") == lists
    fake.fake_fail_malloc(nth)
    with pytest.raises(vfs.VfsError):
        ctx.ibm_search(*cases.icosphere((1.5, 1.0, 3.0), 0.4, 1))
    fake.fake_fail_malloc(0)
    assert fake.fake_launches(b"k_ibm_cast") == 1
    ctx.formfunction2(1.0)
    assert fake.fake_launches(b"k_collect_points") > lists
    ctx.poisson_rhs()
    assert fake.fake_launches(b"k_poisson_coef") > operators
    ctx.close()


@pytest.mark.parametrize("nth", [2, 3, 4, 5])
def test_marks_after_a_search_that_failed_half_way(fake, nth):
    """The search marks cells in Contra2Cart's flag buffer: cleared again on every way out."""
    ctx = context(immersed=1)
    surface = cases.icosphere((1.5, 1.0, 3.0), 0.4, 1)
    ctx.ibm_search(*surface)
    n = ctx.shape[0] * ctx.shape[1] * ctx.shape[2]
    fake.fake_fail_malloc(nth)
    n0 = fake.fake_cleared_bytes()
    with pytest.raises(vfs.VfsError):
        ctx.ibm_search(*surface)
    assert fake.fake_cleared_bytes() - n0 >= n
    ctx.close()
