"""The even-odd cluster kernel stops the Schur solve where the grid-wide one does, so
that which kernel a lattice gets does not decide the error of its propagators.

The grid-wide kernel ends at the first multiple of 16 iterations at which the FP64
residual meets the tolerance, the cluster kernel at the first iteration: 0 to 15
earlier, give or take the few that FP32 iterations differ by, so fewer than 16 in the
mean. A stop at twice the tolerance comes 15 iterations earlier still at this lattice.

The errors against a solve to 1e-13: the residual falls by 2 in 15 iterations, so the
cluster kernel's may be 2 times the grid-wide kernel's, 2.5 with a quarter to spare."""
import numpy as np
import pytest

from conftest import quenched_theta, rel

pytestmark = pytest.mark.gpu


def test_cluster_kernel_is_as_accurate_as_the_grid_kernel():
    import three_part_dwf_study_b200 as T
    from three_part_dwf_study_b200 import _capi as A
    Nt, Nx, Ls, n = 62, 94, 16, 8
    rng = np.random.default_rng(41)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.05)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    src = np.zeros((n, Ls, Nt, Nx, 2), np.complex128)
    for k in range(n):
        src[k, 0, :, :, 1] = rng.choice([1, 1j, -1, -1j], size=(Nt, Nx))
        src[k, Ls - 1, :, :, 0] = rng.choice([1, 1j, -1, -1j], size=(Nt, Nx))
    src = src.reshape(n, -1)

    def solve(rtol, kernel):
        A.check(A.lib().dwf_set_eo_kernel(d.handle, kernel), d.handle)
        n0 = d.solver_kernel_ms(2)[1]
        x, info = d.propagators(src, rtol=rtol, maxiter=20000, solver=T.SOLVER_EO_MIXED)
        assert all(i["converged"] for i in info)
        assert (d.solver_kernel_ms(2)[1] > n0) == (kernel != 0)
        return x, [i["schur_iterations"] for i in info]

    exact, _ = solve(1e-13, -1)
    err, its = {}, {}
    for k in (-1, 0):
        x, it = solve(1e-11, k)
        err[k], its[k] = np.mean([rel(a, b) for a, b in zip(x, exact)]), np.array(it)
    assert (its[0] - its[-1]).mean() < 16, (its[0], its[-1])
    assert err[-1] < 2.5 * err[0], err
    d.close()
