"""Batched and single CG on lattices small enough for one thread-block cluster
per right-hand side, over the shapes the kernel distinguishes: slices that do
not fill a site's threads, rows that do not divide among the CTAs, a last warp
with idle lanes, one CTA, more right-hand sides than resident clusters,
several configurations, a starting guess.

Each solution's residual is recomputed with the operator (1e-13 by other
tests): FP64 CG stops on the recursive residual at 1e-10, at most a few
thousand roundings of |A| |x| (1e-11 of |b|) from the true one; the mixed form
stops on the FP64 true residual."""
import numpy as np
import pytest

from conftest import quenched_theta

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import three_part_dwf_study_b200 as T
    return T


def solve_and_check(T, d, rng, n, nconf, guess, eigen):
    torch = pytest.importorskip("torch")
    d.set_gauge(np.stack([quenched_theta(rng, d.Nt, d.Nx, 3.0) for _ in range(nconf)]))
    conf = np.arange(n) % nconf
    b = torch.from_numpy(rng.normal(size=(n, d.Ndof)) + 1j * rng.normal(size=(n, d.Ndof))).cuda()
    for op in (T.OP_DDDAG, T.OP_DDAGD):
        for solver, tol in ((T.SOLVER_CG64, 1.2e-10), (T.SOLVER_MIXED, 1.001e-10)):
            x = 0.1 * torch.flip(b, dims=[1]) if guess else torch.empty_like(b)
            info = d.cg_batch_dev(op, b, x, rhs_conf=conf, has_guess=guess, rtol=1e-10, maxiter=4000,
                                  solver=solver)
            assert all(i["converged"] and not i["fallback"] for i in info)
            for k in range(n):
                y = torch.empty_like(b[k])
                d.apply_dev(op, x[k], y, conf=int(conf[k]))
                assert float((y - b[k]).norm() / b[k].norm()) < tol, (op, solver, k)


@pytest.mark.parametrize("guess", [False, True])
@pytest.mark.parametrize("Nt,Nx,Ls,n,nconf", [
    (2, 2, 2, 3, 1), (3, 5, 1, 2, 2), (5, 3, 7, 2, 1), (17, 23, 4, 5, 2), (33, 9, 6, 3, 1), (12, 10, 13, 4, 3),
    (8, 8, 4, 300, 5), (31, 16, 24, 2, 1), (40, 40, 8, 1, 1)])
def test_dwf_batches(T, Nt, Nx, Ls, n, nconf, guess):
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1)
    solve_and_check(T, d, np.random.default_rng(Nt * 1000 + Nx * 10 + Ls), n, nconf, guess, False)
    d.close()


@pytest.mark.parametrize("Nt,Nx,n", [(2, 3, 2), (16, 1, 1), (7, 33, 3), (48, 40, 16), (64, 64, 2), (9, 8, 400)])
def test_wilson_batches(T, Nt, Nx, n):
    w = T.Wilson(Nt, Nx, 0.2, bc_t=-1.0, bc_x=1.0)
    solve_and_check(T, w, np.random.default_rng(Nt * 1000 + Nx), n, 2, False, True)
    w.close()


def test_iteration_limit_and_zero_source(T):
    """A limit short of convergence: the mixed solve and its FP64 continuation
    stop there; a zero right-hand side beside it is left at zero."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(8)
    d = T.DomainWall(12, 10, 6, 1.0, 0.05)
    d.set_gauge(quenched_theta(rng, 12, 10, 3.0))
    b = torch.zeros(2, d.Ndof, dtype=torch.complex128, device="cuda")
    b[1] = torch.from_numpy(rng.normal(size=d.Ndof) + 0j).cuda()
    for solver, its in ((T.SOLVER_CG64, 5), (T.SOLVER_MIXED, 10)):
        x = torch.empty_like(b)
        info = d.cg_batch_dev(T.OP_DDDAG, b, x, rtol=1e-10, maxiter=5, solver=solver)
        assert info[0]["converged"] and info[0]["iterations"] == 0 and not bool(x[0].abs().any())
        assert not info[1]["converged"] and info[1]["iterations"] == its
    d.close()
