"""The weight-gradient kernel at channel counts that do not fill its 4 x 4 tiles,
at every number of threads per tile it uses, with sites that do not fill its
chunks of 16. Bars as in test_loss_and_gradient_match_oracle: the oracle's
rounded network within 2e-3 (rare BF16 ties flipped by FP32 rounding of the
intermediate fields), the loss within 1e-5."""
import numpy as np
import pytest

from conftest import quenched_theta, rel
from oracle import learned as LN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls,hidden,Nt,Nx,n", [(1, 8, 5, 7, 3), (3, 8, 9, 6, 2), (5, 24, 4, 11, 2),
                                             (7, 16, 6, 5, 1), (16, 32, 3, 10, 2), (23, 32, 4, 4, 1)])
def test_gradient_at_ragged_channels(Ls, hidden, Nt, Nx, n):
    torch = pytest.importorskip("torch")
    import three_part_dwf_study_b200 as T
    rng = np.random.default_rng(Ls * 100 + hidden)
    d = T.DomainWall(Nt, Nx, Ls, 1.0, 0.05)
    d.set_gauge(quenched_theta(rng, Nt, Nx, 3.0))
    d.lp_init(hidden=hidden, seed=3)
    ws = d.lp_weights()
    V, C0 = Nt * Nx, 2 * Ls

    def field():
        return (rng.normal(size=(n, d.Ndof)) + 1j * rng.normal(size=(n, d.Ndof))).astype(np.complex64)

    rho, e = field(), field()
    loss, grads = d.lp_loss_grad_dev(torch.from_numpy(rho).cuda(), torch.from_numpy(e).cuda())
    Tg = d.lp_transports(0).astype(np.complex128)
    lo, go = LN.loss_grad(Tg, LN.neighbours(Nt, Nx), ws, LN.to_net(rho, V, C0), LN.to_net(e, V, C0), rounded=True)
    assert abs(loss - lo) < 1e-5 * abs(lo)
    for l in range(4):
        assert rel(grads[l], go[l]) < 2e-3, l
    d.close()
