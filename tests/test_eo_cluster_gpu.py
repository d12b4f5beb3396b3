"""The even-odd cluster solver over the shapes its work split distinguishes:
Ls that does not fill the threads of a site, rows that do not divide among the
CTAs, CTAs with one row, one CTA per right-hand side, extents that leave lanes
of the last warp idle, two and four threads per site, e in registers and in
shared memory, more right-hand sides than resident clusters.

Each batch is solved by the FP64 CG on the full lattice too (no shared code).
Both must meet the FP64 stopping rule at 1e-10; two solutions of D^dag D x = b
that meet it differ by at most 2 cond(D^dag D) 1e-10, below 1e-6 at these
masses. The Schur complement's condition is no worse than D's, so its iterations
exceed the FP64 CG's by no more than the reliable updates' restarts (8).
(The grid-wide even-odd kernel is no reference at the smallest lattices: at 4x2x1
CG ends before its first reliable update and it runs to its iteration limit.)"""
import numpy as np
import pytest

from conftest import quenched_theta, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import three_part_dwf_study_b200 as T
    return T


def sources(rng, n, Nt, Nx, Ls):
    v = np.zeros((n, Ls, Nt, Nx, 2), np.complex128)
    for k in range(n):
        if k % 2:
            v[k, 0, :, :, 1] = rng.choice([1, 1j, -1, -1j], size=(Nt, Nx))
            v[k, Ls - 1, :, :, 0] = rng.choice([1, 1j, -1, -1j], size=(Nt, Nx))
        else:
            b = (k // 2) % 2
            v[k, 0 if b else Ls - 1, (k * 3) % Nt, (k * 5) % Nx, b] = 1.0
    return v.reshape(n, -1)


@pytest.mark.parametrize("Nt,Nx,Ls,n", [
    (2, 2, 2, 1), (4, 2, 1, 3), (8, 6, 3, 2), (10, 14, 5, 3), (18, 10, 6, 4), (34, 22, 7, 2),
    (12, 8, 10, 200), (46, 18, 13, 3), (16, 40, 15, 2), (64, 96, 16, 3), (62, 94, 16, 2), (24, 20, 18, 9),
    (32, 16, 24, 5), (30, 34, 23, 2)])
def test_cluster_solver_matches_fp64_cg(T, Nt, Nx, Ls, n):
    rng = np.random.default_rng(Nt * 10000 + Nx * 100 + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    src = sources(rng, n, Nt, Nx, Ls)
    n0 = d.solver_kernel_ms(2)[1]
    x, info = d.propagators(src, rtol=1e-10, maxiter=20000, solver=T.SOLVER_EO_MIXED)
    assert d.solver_kernel_ms(2)[1] > n0  # the cluster kernel ran
    y, jnfo = d.propagators(src, rtol=1e-10, maxiter=20000, solver=T.SOLVER_CG64)
    for k in range(n):
        assert info[k]["converged"] and info[k]["true_relres"] <= 1e-10, k
        assert jnfo[k]["converged"] and jnfo[k]["true_relres"] <= 1.2e-10, k
        assert info[k]["schur_iterations"] <= jnfo[k]["iterations"] + 8, k
        assert rel(x[k], y[k]) < 1e-6, k
    d.close()


def test_cluster_solver_stops_at_its_iteration_limit(T):
    """maxiter short of convergence: every right-hand side stops there."""
    rng = np.random.default_rng(5)
    d = T.DomainWall(24, 20, 8, 1.0, 0.05)
    d.set_gauge(quenched_theta(rng, 24, 20, 3.0))
    src = sources(rng, 3, 24, 20, 8)
    _, info = d.propagators(src, rtol=1e-10, maxiter=7, solver=T.SOLVER_EO_MIXED)
    assert all(i["schur_iterations"] == 7 and not i["converged"] for i in info)
    d.close()
