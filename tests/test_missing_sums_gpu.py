"""Waits that run out inside the solvers that exchange sums by messages: one block
waits for a sum that is never sent, the others then for what that block no longer
sends, every block leaves on its own, the call reports DWF_TIMEOUT and the context solves as before.

The cases are the places a wait can end differently in different CTAs of a cluster:
the first sum of a right-hand side, the middle of an iteration, and the sum that
sends all CTAs but one into a reliable update (maxiter = 1: the first iteration asks
for one) or to the end of the right-hand side; clusters of one and of sixteen CTAs, and
more right-hand sides than resident clusters.

A mixed solve that gives up ends at once: nothing to compare but its status. The solve
after it has to give the bits of the one before (fixed orders of all sums)."""
import numpy as np
import pytest

from conftest import quenched_theta

pytestmark = pytest.mark.gpu

LIMIT = 20_000_000  # ns; a solve here takes a few milliseconds


@pytest.fixture(scope="module")
def T():
    import three_part_dwf_study_b200 as T
    return T


def check(d, solve, masks):
    from three_part_dwf_study_b200 import _capi as A
    before = solve(3000)
    for mask in masks:
        for maxiter in (3000, 1):
            A.check(A.lib().dwf_set_wait_limit(d.handle, LIMIT), d.handle)
            A.check(A.lib().dwf_set_missing_sums(d.handle, mask), d.handle)
            with pytest.raises(RuntimeError, match="ran out"):
                solve(maxiter)
            A.check(A.lib().dwf_set_missing_sums(d.handle, 0), d.handle)
            A.check(A.lib().dwf_set_wait_limit(d.handle, 5_000_000_000), d.handle)
            assert np.array_equal(solve(3000), before), (mask, maxiter)


def sources(rng, n, d):
    return rng.normal(size=(n, d.Ndof)) + 1j * rng.normal(size=(n, d.Ndof))


@pytest.mark.parametrize("Nt,Nx,Ls,n", [(16, 12, 8, 3), (64, 32, 16, 20), (2, 4, 2, 2)])
def test_even_odd_cluster_solver(T, Nt, Nx, Ls, n):
    rng = np.random.default_rng(Nt + Nx + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    src = sources(rng, n, d)
    k0 = d.solver_kernel_ms(2)[1]
    check(d, lambda m: d.propagators(src, rtol=1e-8, maxiter=m, solver=T.SOLVER_EO_MIXED)[0], (1, 2, 4))
    assert d.solver_kernel_ms(2)[1] > k0  # the cluster kernel ran
    d.close()


@pytest.mark.parametrize("solver", ["SOLVER_CG64", "SOLVER_MIXED"])
@pytest.mark.parametrize("Nt,Nx,Ls,n", [(16, 12, 4, 3), (48, 40, 1, 9), (2, 3, 2, 2), (64, 64, 16, 1), (2, 2, 25, 1)])
def test_full_lattice_solvers(T, Nt, Nx, Ls, n, solver):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(Nt + Nx + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1) if Ls > 1 else T.Wilson(Nt, Nx, 0.1)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    b = torch.from_numpy(sources(rng, n, d)).cuda()

    def solve(maxiter):
        x = torch.empty_like(b)
        d.cg_batch_dev(T.OP_DDDAG, b, x, rtol=1e-8, maxiter=maxiter, solver=getattr(T, solver))
        return x.cpu().numpy()

    check(d, solve, (1, 2, 4, 8))
    d.close()


def test_a_limit_that_any_wait_may_exceed(T):
    """With a limit of a nanosecond each wait may run out or not, in any warp: a solve
    converges or gives up, and what follows on the context is as before."""
    from three_part_dwf_study_b200 import _capi as A
    rng = np.random.default_rng(4)
    d = T.DomainWall(24, 20, 6, 1.0, 0.1)
    d.set_gauge(quenched_theta(rng, 24, 20, 3.0))
    src = sources(rng, 9, d)

    def solves():
        return [d.propagators(src, rtol=1e-8, maxiter=3000, solver=s)[0]
                for s in (T.SOLVER_EO_MIXED, T.SOLVER_MIXED, T.SOLVER_CG64)]

    before = solves()
    for _ in range(5):
        A.check(A.lib().dwf_set_wait_limit(d.handle, 1), d.handle)
        try:
            solves()
        except RuntimeError as e:
            assert "ran out" in str(e)
        A.check(A.lib().dwf_set_wait_limit(d.handle, 5_000_000_000), d.handle)
        assert all(np.array_equal(a, b) for a, b in zip(solves(), before))
    d.close()
