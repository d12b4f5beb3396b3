"""Solves of one right-hand side at the sizes where their kernels change shape:
fewer sites than one block, a ragged last block, the largest lattice with one
site per thread and the first without, extents that are not multiples of a warp.

The solver's own claim (the stopping rule at 1e-10) is recomputed with the
operator, which other tests hold to 1e-13: FP64 CG stops on the recursive
residual, whose distance from the true one is at most a few thousand roundings
of |A| |x| (1e-11 of |b| here), the mixed form on the FP64 true residual. Both
solutions are within cond(D D^dag) * 1e-10 < 1e-6 of the exact one."""
import numpy as np
import pytest

from conftest import quenched_theta, random_field, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import three_part_dwf_study_b200 as T
    return T


@pytest.mark.parametrize("guess", [False, True])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 1), (8, 8, 2), (13, 37, 3), (17, 31, 9),
                                   (64, 64, 18), (64, 64, 19), (50, 70, 24)])
def test_single_solve_meets_its_rule(T, shape, guess):
    Nt, Nx, Ls = shape
    rng = np.random.default_rng(Nt * 1000 + Nx * 10 + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1)
    th = quenched_theta(rng, Nt, Nx, 3.0)
    b = random_field(rng, d.Ndof)
    x0 = 0.1 * random_field(rng, d.Ndof) if guess else None
    xs = []
    for op in (T.OP_DDDAG, T.OP_DDAGD):
        for solver, tol in ((T.SOLVER_CG64, 1.2e-10), (T.SOLVER_MIXED, 1.001e-10)):
            r = d.conjugate_gradient(op, th, b, initial_guess=x0, rtol=1e-10, maxiter=4000, solver=solver)
            assert r.converged and not r.info["fallback"]
            assert rel(d.apply(op, th, r.x), b) < tol
            xs.append(r.x)
    assert rel(xs[1], xs[0]) < 1e-6 and rel(xs[3], xs[2]) < 1e-6
    d.close()


@pytest.mark.parametrize("shape", [(3, 5), (32, 32), (48, 40), (256, 300)])
def test_single_wilson_solve_meets_its_rule(T, shape):
    Nt, Nx = shape
    rng = np.random.default_rng(Nt * 1000 + Nx)
    w = T.Wilson(Nt, Nx, 0.2, bc_t=-1.0, bc_x=1.0)
    th = quenched_theta(rng, Nt, Nx, 3.0)
    b = random_field(rng, w.Ndof)
    for solver, tol in ((T.SOLVER_CG64, 1.2e-10), (T.SOLVER_MIXED, 1.001e-10)):
        r = w.conjugate_gradient(T.OP_DDDAG, th, b, rtol=1e-10, maxiter=4000, solver=solver)
        assert r.converged and rel(w.apply(T.OP_DDDAG, th, r.x), b) < tol
    w.close()
