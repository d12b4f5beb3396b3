"""The full-lattice kernels that the shapes of other tests do not reach, since lattices
that fit a thread-block cluster run there: the batch kernels (bits of repeated solves,
which a sum read while another block stores into its slot breaks about once in a
thousand) and the whole-GPU kernel of one right-hand side with fewer sites than one
block. And Eigen's iteration count from the cluster kernel.

A lattice does not fit a cluster when no split into 16 CTAs at most and 8 threads a site
leaves a thread at most 3 (FP64) or 6 (mixed) slices, a CTA 512 threads, and p and t with
a halo row either side 227 KB."""
import numpy as np
import pytest

from conftest import quenched_theta, random_field, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import three_part_dwf_study_b200 as T
    return T


def fits_cluster(Nt, Nx, Ls, mixed):
    for R in range(1, Nt + 1):
        for NL in (1, 2, 4, 8):
            threads = -(-R * Nx // (32 // NL)) * 32
            if (-(-Nt // R) <= 16 and -(-Ls // NL) <= (6 if mixed else 3) and threads <= 512
                    and 2 * Ls * (R + 2) * Nx * (16 if mixed else 32) <= 227 * 1024):
                return True
    return False


@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("Nt,Nx,Ls,n", [(64, 64, 16, 3), (5, 3, 49, 2)])
def test_repeated_batches_are_bit_identical(T, Nt, Nx, Ls, n, solver):
    torch = pytest.importorskip("torch")
    assert not fits_cluster(Nt, Nx, Ls, solver == 1)
    rng = np.random.default_rng(Nt + Nx + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.2)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    b = torch.from_numpy(rng.normal(size=(n, d.Ndof)) + 1j * rng.normal(size=(n, d.Ndof))).cuda()
    x0, x = torch.empty_like(b), torch.empty_like(b)
    d.cg_batch_dev(T.OP_DDDAG, b, x0, rtol=1e-6, maxiter=3000, solver=solver)
    for _ in range(150):
        d.cg_batch_dev(T.OP_DDDAG, b, x, rtol=1e-6, maxiter=3000, solver=solver)
        assert torch.equal(torch.view_as_real(x), torch.view_as_real(x0))
    d.close()


@pytest.mark.parametrize("guess", [False, True])
@pytest.mark.parametrize("shape,solver", [((3, 5, 49), 0), ((3, 5, 49), 1), ((2, 2, 25), 0), ((1, 7, 50), 1),
                                          ((11, 13, 53), 0), ((11, 13, 53), 1)])
def test_one_right_hand_side_on_few_sites(T, shape, solver, guess):
    """Bars as in test_single_solve_gpu.py."""
    Nt, Nx, Ls = shape
    assert not fits_cluster(Nt, Nx, Ls, solver == 1)
    rng = np.random.default_rng(Nt * 1000 + Nx * 10 + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1)
    th = quenched_theta(rng, Nt, Nx, 3.0)
    b = random_field(rng, d.Ndof)
    x0 = 0.1 * random_field(rng, d.Ndof) if guess else None
    for op in (T.OP_DDDAG, T.OP_DDAGD):
        r = d.conjugate_gradient(op, th, b, initial_guess=x0, rtol=1e-10, maxiter=4000, solver=solver)
        assert r.converged and not r.info["fallback"]
        assert rel(d.apply(op, th, r.x), b) < (1.001e-10 if solver else 1.2e-10)
    d.close()


@pytest.mark.parametrize("Nt,Nx", [(16, 12), (7, 33), (32, 32)])
def test_eigen_iteration_count_of_the_cluster_kernel(T, Nt, Nx):
    """solve_CGNR counts as Eigen's ConjugateGradient: the iteration that meets
    |r|^2 < tol^2 |b|^2 is not counted. The same recurrence in numpy, the operator
    applied by the library; 1e-6 is far from rounding."""
    assert fits_cluster(Nt, Nx, 1, False)
    rng = np.random.default_rng(Nt + Nx)
    w = T.Wilson(Nt, Nx, 0.2, bc_t=-1.0, bc_x=1.0)
    th = quenched_theta(rng, Nt, Nx, 3.0)
    src = random_field(rng, w.Ndof)
    b = w.apply(T.OP_DDAG, th, src)
    r, p, n = b.copy(), b.copy(), 0
    while True:
        ap = w.apply(T.OP_DDAGD, th, p)
        rr = np.vdot(r, r).real
        r = r - rr / np.vdot(p, ap).real * ap
        rn = np.vdot(r, r).real
        if rn < 1e-12 * np.vdot(b, b).real:
            break
        p, n = r + rn / rr * p, n + 1
    assert w.solve_CGNR(th, src, 1e-6, 4000)["iterations"] == n > 5
    w.close()
