"""Device entry points called with torch's current stream other than the default
one: what the stream was still computing is the input, and what the stream does
next sees the output. The producer runs behind a wait of some 10 ms on the device, so a
call that ran ahead of it, or a reader that ran ahead of the call, would see the
buffers' earlier contents (zeros). The same for dwf_stream_enter / _leave with NULL, the
device's default stream."""
import numpy as np
import pytest

from conftest import quenched_theta

pytestmark = pytest.mark.gpu

WAIT = 20_000_000  # clock cycles


@pytest.fixture(scope="module")
def setup():
    torch = pytest.importorskip("torch")
    import three_part_dwf_study_b200 as T
    rng = np.random.default_rng(11)
    d = T.DomainWall(16, 12, 4, 1.0, 0.2)
    th = quenched_theta(rng, 16, 12, 3.0)
    d.set_gauge(th)
    f = torch.from_numpy(rng.normal(size=(2, d.Ndof)) + 1j * rng.normal(size=(2, d.Ndof))).cuda()
    yield torch, T, d, th, f
    d.close()


def calls(torch, T, d, th, f):
    """name -> (field type, call(in, out))"""
    thd = torch.from_numpy(th).cuda()
    return {
        "apply": (torch.complex128, lambda i, o: d.apply_dev(T.OP_DDAG, i, o)),
        "apply32": (torch.complex64, lambda i, o: d.apply_dev(T.OP_DDAGD, i, o)),
        "set_gauge": (torch.complex128, lambda i, o: (d.set_gauge_dev(thd), d.apply_dev(T.OP_D, i, o))),
        "cg": (torch.complex128, lambda i, o: d.cg_batch_dev(T.OP_DDDAG, i, o, rtol=1e-8, maxiter=2000)),
        "propagators": (torch.complex128, lambda i, o: d.propagators_dev(i, o, rtol=1e-8, maxiter=2000,
                                                                          solver=T.SOLVER_EO_MIXED)),
    }


@pytest.mark.parametrize("name", ["apply", "apply32", "set_gauge", "cg", "propagators"])
def test_call_on_a_side_stream(setup, name):
    torch, T, d, th, f = setup
    dtype, call = calls(torch, T, d, th, f)[name]
    f = f.to(dtype)
    want = torch.zeros_like(f)
    call(f, want)
    call(f, want)  # tuned, workspaces there
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    i, o, seen = (torch.zeros_like(f) for _ in range(3))
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(WAIT)
        i.copy_(f)
        call(i, o)
        seen.copy_(o)
    s.synchronize()
    assert torch.equal(torch.view_as_real(seen), torch.view_as_real(want))


def test_enter_and_leave_the_default_stream(setup):
    import ctypes as C
    torch, T, d, th, f = setup
    from three_part_dwf_study_b200 import _capi as A
    want, i, o, seen = (torch.zeros_like(f) for _ in range(4))
    d.apply_dev(T.OP_D, f, want)
    torch.cuda.synchronize()
    torch.cuda._sleep(WAIT)
    i.copy_(f)
    A.check(A.lib().dwf_stream_enter(d.handle, None), d.handle)
    A.check(A.lib().dwf_apply_dev(d.handle, T.OP_D, 0, C.c_void_p(i.data_ptr()), C.c_void_p(o.data_ptr()), 2, 64),
            d.handle)
    A.check(A.lib().dwf_stream_leave(d.handle, None), d.handle)
    seen.copy_(o)
    torch.cuda.synchronize()
    assert torch.equal(torch.view_as_real(seen), torch.view_as_real(want))
