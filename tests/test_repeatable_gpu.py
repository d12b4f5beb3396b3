"""The persistent solvers add in fixed orders and decide on the same bits in
every block, so a repeated solve gives the same bits. A block that read a partial
sum another block had already overwritten broke that about once in a thousand
solves (and could leave a solution off by what one wrong step length does); 150
repetitions of each kernel are a guard, not a proof."""
import numpy as np
import pytest

from conftest import quenched_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nt,Nx,Ls,n", [(32, 32, 1, 1), (16, 12, 8, 9), (40, 42, 12, 3), (48, 48, 16, 1)])
@pytest.mark.parametrize("solver", [0, 1])
def test_repeated_solves_are_bit_identical(Nt, Nx, Ls, n, solver):
    torch = pytest.importorskip("torch")
    import three_part_dwf_study_b200 as T
    rng = np.random.default_rng(Nt + Nx + Ls)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.1) if Ls > 1 else T.Wilson(Nt, Nx, 0.1)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    b = torch.from_numpy(rng.normal(size=(n, d.Ndof)) + 1j * rng.normal(size=(n, d.Ndof))).cuda()
    x0, x = torch.empty_like(b), torch.empty_like(b)
    d.cg_batch_dev(T.OP_DDDAG, b, x0, rtol=1e-6, maxiter=3000, solver=solver)
    for _ in range(150):
        d.cg_batch_dev(T.OP_DDDAG, b, x, rtol=1e-6, maxiter=3000, solver=solver)
        assert torch.equal(torch.view_as_real(x), torch.view_as_real(x0))
    d.close()
